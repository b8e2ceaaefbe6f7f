// experts_mma.cu - decode-sized grouped experts for NVFP4 and IQ3_S blobs: a bandwidth-bound weight stream through shared memory
// with the dot products on the tensor cores.
//
// Shape of the work (HBM-bound): every touched expert's gate, up and down rows are read exactly once per pass of up to 8
// activation columns.  Each warp owns 16 weight rows (8 gate rows paired with the 8 matching up rows, or 16 down rows) and
// streams them in 256-column chunks (144 bytes a row) through its own cp.async ring of two or three stages, so no block-wide barrier
// sits in the stream.  A row's E2M1 codes go to fp16 pairs with cvt.rn.f16x2.e2m1x2 (one ALU-pipe
// instruction per byte, the scarce resource here: the ALU pipe issues at half rate), are multiplied by the block's UE4M3
// scale as fp16 (the product has at most 5 significant bits: exact; the scale comes from a 256-entry shared-memory table)
// and feed mma.sync.m16n8k16 with fp32 accumulation.  Each of a row group's four threads owns one 16-value sub-block, so it
// decodes one scale per row and block.  The activation columns (8 bf16 tokens, or 4 fp32 tokens split into hi + lo fp16
// terms, each row pre-scaled by a power of two so it fits fp16) are prepared once per call by a small kernel into
// B-fragment order and copied into shared memory by cp.async.  Gate and up rows of one neuron land in the same thread's
// accumulators, so SwiGLU is fused; a second small kernel turns the SwiGLU output into the down product's fp16 image.
//
// IQ3_S rows take the same stream with another decoder (iq3s_16): codebook points as four fp16 magnitudes in shared memory, signs
// and the odd scales applied in packed fp16, exactly.  Bound by the decode's integer work and look-ups.
//
// What the launch shape is worth (equal runs of row blocks, sixteen warps an SM, whole-row or split tiles: launch() below), 2048 x 512 unless
// said: IQ3_S, 512 experts, 5 tokens 125 -> 99 us, 64 tokens 420 -> 305; NVFP4, 1 token 52 -> 34, 64 tokens 169 -> 154, 27 tokens of
// 2560 x 640 223 -> 175.
//
// IQ1_M rows take it where the integer kernel (experts_kq.cu) does not: widths of an odd number of 256-column blocks, which the
// warp-per-row fp32 kernels had before, so the results may be no further off than theirs.  Weights are 8 w / d, exact in fp16 (iq1m.cuh);
// a row is two fp16 terms, which costs one rounding of 2^-24 a value and what lies below 2^-38 of the row's largest, against the fp32
// kernels' longer chains.  A row's distance to 64-bit sums (root mean square over rows), fp32 kernels and this one: 5120 x 2304 normal fp32
// rows 3.8e-7 and 1.9e-7, bf16 3.8e-7 and 1.5e-7, rows of a few large values (lognormal, sigma 4) 3.1e-7 and 2.0e-7; 1280 x 1280 2.4e-7 and
// 1.7e-7, 2.4e-7 and 1.4e-7, 2.1e-7 and 1.9e-7; the narrowest, 256 x 256, 2.1e-7 and 1.6e-7, 2.1e-7 and 1.3e-7, 1.78e-7 and 1.82e-7.
//
// Semantics: Basalt's native_expert_grouped (include/basalt/kernels/iq_kernels.hpp:77-92; kernels src/kernels/cuda/iq_kernels.cu:
// 1605-1658 gate/up, :2512-2524 SwiGLU, :2140-2164 down), NVFP4 decoding per src/kernels/cpu/ggml/ggml_quants.c:1397-1422,
// tail scales per iq_kernels.cu:683-701 - but without the int8 rounding of x and h the reference applies.
#include <atomic>
#include <cuda_fp16.h>

#include "common.cuh"
#include "experts.cuh"
#include "formats.cuh"
#include "iq1m.cuh"
#include "pdl.cuh"
#include "plan.cuh"

namespace bsx {
namespace {

constexpr int kRows = 16;                      // weight rows per warp
constexpr int kCols = 8;                       // MMA n: activation columns per pass

// The formats.  A chunk of a row is what a stage holds: 4 NVFP4 blocks of 64 columns, 2 IQ3_S blocks of 256 (110 bytes, so every
// second one starts on 4 bytes) or 2 IQ1_M blocks of 256 (56 bytes; a row may end in one).  kTable: the shared-memory table, 256 fp16 scale
// pairs, 512 points of four fp16 magnitudes or the 2048 points of the IQ1 codebook as they are.
enum { FMT_NVFP4 = 0, FMT_IQ3S = 1, FMT_IQ1M = 2 };
template <int FMT> struct Fmt;
template <> struct Fmt<FMT_NVFP4> {
    static constexpr int kRowBytes = 144, kGranules = 4, kTable = 1024;
    static constexpr float kUnscale = 256.f;           // the block scales are used as scale / 2^8
};
template <> struct Fmt<FMT_IQ3S> {
    static constexpr int kRowBytes = 220, kGranules = 8, kTable = 4096;
    static constexpr float kUnscale = 1.f;
};
template <> struct Fmt<FMT_IQ1M> {
    static constexpr int kRowBytes = 112, kGranules = 8, kTable = 4096;
    static constexpr float kUnscale = 0.125f;          // weights enter as 8 w / d
};
template <int FMT> constexpr int kStageBytes = kRows * Fmt<FMT>::kRowBytes;

enum { MODE_GU = 0, MODE_DOWN = 1 };

__device__ __forceinline__ void cp_async16(uint32_t smem_addr, const void* gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(smem_addr), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int BYTES>
__device__ __forceinline__ void cp_async_piece(uint32_t smem_addr, const void* gmem) {   // BYTES 16, 8 or 4, both addresses aligned to it
    if constexpr (BYTES == 16) cp_async16(smem_addr, gmem);
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(smem_addr), "l"(gmem), "n"(BYTES) : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// four E2M1 pairs (one byte each) of a 32-bit word -> four fp16 pairs; low nibble in the low half
__device__ __forceinline__ void cvt_e2m1x8(uint32_t w, uint32_t (&h)[4]) {
    asm("{\n"
        ".reg .b8 b0, b1, b2, b3;\n"
        "mov.b32 {b0, b1, b2, b3}, %4;\n"
        "cvt.rn.f16x2.e2m1x2 %0, b0;\n"
        "cvt.rn.f16x2.e2m1x2 %1, b1;\n"
        "cvt.rn.f16x2.e2m1x2 %2, b2;\n"
        "cvt.rn.f16x2.e2m1x2 %3, b3;\n"
        "}\n"
        : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
        : "r"(w));
}

__device__ __forceinline__ uint32_t hmul2_bits(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma_f16_zero(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};\n"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

// UE4M3 scale byte -> fp16 pair {d, d} with d = scale / 2^8: (byte & 0x7F) << 7 puts E4M3's exponent and mantissa where
// fp16 keeps them (value 2^(e-15) (1 + m/8), subnormals included) while the scale itself is 2^(e-7) (1 + m/8) (ggml halves
// it only because its E2M1 table is doubled; the cvt above yields undoubled values), so the epilogue multiplies the sums
// by 2^8.  0x7F decodes to 0 and bit 7 is ignored (src/kernels/cpu/ggml/ggml_quants.c:1397-1406).
__device__ __forceinline__ uint32_t scale_pair_bits(uint32_t byte) {
    const uint32_t b = byte & 0x7Fu;
    const uint32_t v = b == 0x7Fu ? 0u : b << 7;
    return v | (v << 16);
}

// IQ3_S (include/basalt/ggml/ggml_common.h block_iq3_s: fp16 d, qs[64], qh[8], signs[32], scales[4]; decode rule
// src/kernels/cpu/ggml/ggml_quants.c:1200-1239): a weight is d (2 s + 1) x +-(2 c + 1), c a 3-bit coordinate of a 512-point
// codebook.  One thread decodes the 16 values [16 t, 16 t + 16) of granule `gr` (64 columns) of a row's block: four points, 16 sign
// bits, one scale.  Magnitude x scale is an integer up to 465, exact in fp16; d stays outside the sums.  q[i]: values 2 i and 2 i + 1,
// as a point holds them.  points: the lane's copy of the codebook, NC copies interleaved point by point.
template <int NC>
__device__ __forceinline__ void iq3s_16(const uint8_t* blk, int gr, int t, const uint2* __restrict__ points, uint32_t (&q)[8]) {
    const int ib = 2 * gr + (t >> 1), half = t & 1;
    const uint16_t* qs = reinterpret_cast<const uint16_t*>(blk + 2 + 8 * ib + 4 * half);
    const uint32_t q01 = qs[0], q23 = qs[1];
    const uint32_t qh = (uint32_t) blk[66 + ib] >> (4 * half);
    const uint32_t sg = *reinterpret_cast<const uint16_t*>(blk + 74 + 4 * ib + 2 * half);
    const uint32_t s = ((uint32_t) blk[106 + gr] >> (4 * (t >> 1))) & 15u;      // 2 units of 32 columns a byte
    // 2 s + 1 as an fp16 pair: 1024 + (2 s + 1) is a fp16 whose low bits are the integer
    const __half2 m = __hsub2(__halves2half2(__ushort_as_half((unsigned short) (0x6400u + 2u * s + 1u)), __ushort_as_half((unsigned short) (0x6400u + 2u * s + 1u))),
                              __float2half2_rn(1024.f));
    const uint32_t mm = *reinterpret_cast<const uint32_t*>(&m);
    const uint2 p0 = points[((q01 & 0xFFu) | ((qh & 1u) << 8)) * NC], p1 = points[((q01 >> 8) | ((qh & 2u) << 7)) * NC];
    const uint2 p2 = points[((q23 & 0xFFu) | ((qh & 4u) << 6)) * NC], p3 = points[((q23 >> 8) | ((qh & 8u) << 5)) * NC];
    const uint32_t sw = sg | (sg << 15);                                         // signs 2 i at bit 2 i, signs 2 i + 1 sixteen above
    const uint32_t v[8] = {p0.x, p0.y, p1.x, p1.y, p2.x, p2.y, p3.x, p3.y};
#pragma unroll
    for (int i = 0; i < 8; ++i) q[i] = hmul2_bits(v[i] ^ ((sw << (15 - 2 * i)) & 0x80008000u), mm);
}

// An activation row's fp16 image is laid out so that a thread's B fragments are two 16-byte pieces per 64 columns: piece (gran, h, t)
// holds, for sub-block t of granule gran, the values the thread with id-in-group t needs for MMA steps 2h and 2h + 1.  NVFP4: step s
// takes code bytes 2s and 2s + 1 of the sub-block's 8 bytes; byte b holds values b (low nibble -> k slot 2t) and b + 8 (high nibble ->
// k slot 2t + 1), bytes 2s + 1 go to slots 2t + 8, 2t + 9.  IQ3_S: the values in order (points hold neighbours).

__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    return (uint32_t) __half_as_ushort(__float2half_rn(lo)) | ((uint32_t) __half_as_ushort(__float2half_rn(hi)) << 16);
}

// One warp per activation row: the row -> fp16 image(s) in fragment order plus the inverse of the power of two it was
// scaled by, so that its largest finite magnitude lands in [2^13, 2^14): inside fp16 and with all its bits for every fp32 row
// (2^149 is the largest scale; it makes a row of nothing but the smallest numbers integers below 2^23, which the two terms hold
// exactly; a value below 2^-38 of its row's largest is lost).  An infinity is the first term alone: it reaches the sums as in fp32
// and leaves the row's other values theirs.  A lane takes one 16-value sub-block at a time, which is exactly two 16-byte pieces of
// the image (see image_index).
// FROM_H = false: rows of x (kind x_kind, width n_embd) - row i of x when the caller gave the number of x rows, else the
// row of entry i; true: row e of the SwiGLU output h (fp32, width n_ff).
// The last block lists the passes of the product that follows: a pass is up to 8 / TERMS consecutive entries of one group,
// items[i] = {blob, first entry, entries}, so that kernel's blocks take passes however the entries are spread.
template <int FMT, bool FROM_H, int TERMS>
__global__ void __launch_bounds__(256)
prep_image_kernel(ExpertArgs a, __half* __restrict__ img, float* __restrict__ inv, PassRec* __restrict__ items, int* __restrict__ n_items) {
    pdl_wait();
    pdl_launch_dependents();
    const int ng = min(*a.n_groups, (int) a.cap_groups);
    const int total = min(a.grp_start[ng], (int) a.cap_entries);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (blockIdx.x == gridDim.x - 1) {
        constexpr int NTOK = kCols / TERMS;
        __shared__ int sh[8];
        __shared__ int s_base;
        if (threadIdx.x == 0) s_base = 0;
        __syncthreads();
        for (int g0 = 0; g0 < ng; g0 += 256) {
            const int g = g0 + threadIdx.x;
            const int s0 = g < ng ? a.grp_start[g] : 0;
            const int cnt = g < ng ? max(0, min(a.grp_start[g + 1], (int) a.cap_entries) - s0) : 0;
            const int np = (cnt + NTOK - 1) / NTOK;
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
                r.eb = s0 + p * NTOK;
                r.ntok = min(NTOK, cnt - p * NTOK);
                items[before + x - np + p] = r;
            }
            __syncthreads();
            if (threadIdx.x == 255) s_base = before + x;
            __syncthreads();
        }
        if (threadIdx.x == 0) n_items[0] = s_base;
        return;
    }
    const int i = blockIdx.x * 8 + warp;   // image row
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
        for (int j = 0; j < 16; ++j) amax = fmaxf(amax, isfinite(v[j]) ? fabsf(v[j]) : 0.f);
    }
    amax = warp_max_xor(amax);
    int ex = 0;
    if (amax > 0.f) {
        frexpf(amax, &ex);                          // amax = f 2^ex, f in [0.5, 1)
        ex = min(149, 14 - ex);
    }
    const float s = ldexpf(1.f, min(ex, 100)), s_rest = ldexpf(1.f, max(ex - 100, 0));    // 2^149 is no fp32 number, its inverse is
    if (lane == 0) inv[i] = ldexpf(1.f, -ex);
    uint4* out = reinterpret_cast<uint4*>(img + (size_t) i * K * TERMS);
    for (int sb = lane; sb < n_sb; sb += 32) {
        float v[16];
        load16(src, kind, row, K, sb, v);
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = v[j] * s * s_rest;
        // pieces (gran, 0, t) and (gran, 1, t): values {0,8,1,9,2,10,3,11} and {4,12,5,13,6,14,7,15}, or {0,...,7} and {8,...,15}
        const int piece = ((sb >> 2) * 2) * 4 + (sb & 3);
        auto store = [&](uint4* o, const float (&w)[16]) {
            uint32_t u[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) u[j] = FMT == FMT_IQ3S ? pack_half2(w[2 * j], w[2 * j + 1]) : pack_half2(w[j], w[j + 8]);
            o[piece] = make_uint4(u[0], u[1], u[2], u[3]);
            o[piece + 4] = make_uint4(u[4], u[5], u[6], u[7]);
        };
        store(out, v);
        if (TERMS == 2) {
            float r[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) r[j] = isinf(v[j]) ? 0.f : v[j] - __half2float(__float2half_rn(v[j]));
            store(out + (K >> 3), r);
        }
    }
}

// MODE_GU:  rows = 8 gate rows r0.. paired with up rows r0..; columns = the entries' x images; writes h (fp32).
// MODE_DOWN: rows = 16 down rows; columns = the entries' h images; writes out rows through ent_dst.
// TERMS = 1: 8 entries a pass; TERMS = 2: 4 entries a pass, each as hi + lo fp16 columns.
// PIECE: bytes of one weight copy = the rows' alignment.  16 where K is whole 256-column chunks; a row of any other K (whole
// 64-column NVFP4 blocks, 36 bytes each) starts on 8 bytes (K % 128 == 0) or 4, and its last chunk holds fewer than four blocks:
// those pieces are not requested and those blocks not multiplied.
// CHAIN: MMAs that add up in one accumulator.  The tensor core truncates where it adds to an accumulator, fp32 arithmetic rounds to
// nearest.  Distance to 64-bit sums of the 2048 x 512 layer's fp32 rows: a whole row chained 1.64e-6, 8 MMAs 2.9e-7, 4 (a block of 64
// columns) 2.1e-7, 2 1.8e-7, 1 1.7e-7; the fp32 kernel 2.6e-7.  Its 64-token step, one layer again and again: with four 95 us, with one 98.6.
// Four where no layout needs better.  IQ3_S and NVFP4 with ragged down rows, which the fp32 kernel had before, take one: with four,
// bf16 rows would be further off than there (1.75e-7 against 1.6e-7 at 2560 x 640).
// KS > 1: KS neighbouring warps share a row tile, each a part of its chunks; their sums meet in shared memory.
// Work: the row blocks (W / KS tiles) of all passes in one sequence, cut into equal runs, one a block; a run's part of one pass shares
// its columns and its weight stream.
// W, OCC, ST, NC: warps a block, blocks an SM, stages a warp, copies of the IQ3_S codebook (launch() below).
template <int FMT, int MODE, int TERMS, int PIECE, int CHAIN, int W, int OCC, int ST, int NC, int KS>
__global__ void __launch_bounds__(W * 32, OCC)
blk_mma_kernel(ExpertArgs a, const __half* img, const float* inv, const PassRec* items, const int* n_items, int n_row_blocks) {
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int kThreads = W * 32, kStages = ST, kTiles = W / KS;
    const int64_t K = MODE == MODE_GU ? a.L.n_embd : a.L.n_ff;
    const int n_gran = (int) (K >> 6);                       // 64-column granules
    __half* xs = reinterpret_cast<__half*>(smem);            // [n_gran][2][8 cols][4][8]
    using F = Fmt<FMT>;
    constexpr int kRowBytes = F::kRowBytes, kStageB = kStageBytes<FMT>;
    uint32_t* lut = reinterpret_cast<uint32_t*>(smem + (size_t) K * kCols * 2);     // the format's table
    uint4* zero = reinterpret_cast<uint4*>(smem + (size_t) K * kCols * 2 + F::kTable * NC);   // 64 zero bytes: the B fragments of unused columns
    uint8_t* wbase = smem + (size_t) K * kCols * 2 + F::kTable * NC + 128;
    float4* part = reinterpret_cast<float4*>(wbase + (size_t) W * kStages * kStageB);         // [2][tiles][KS - 1][32] (KS > 1)
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    uint8_t* wring = wbase + (size_t) warp * kStages * kStageB;
    const uint32_t wring_s = (uint32_t) __cvta_generic_to_shared(wring);
    const uint32_t xs_s = (uint32_t) __cvta_generic_to_shared(xs);

    __shared__ int s_ir[kCols];                        // image row of each entry of the pass
    // the first barrier below publishes the table
    if constexpr (FMT == FMT_NVFP4) {
        if (threadIdx.x < 256) lut[threadIdx.x] = scale_pair_bits(threadIdx.x);
    } else if constexpr (FMT == FMT_IQ1M) {
        for (int i = threadIdx.x; i < 1024; i += kThreads) lut[i] = reinterpret_cast<const uint32_t*>(a.grid)[i];
    } else {
        for (int i = threadIdx.x; i < 512 * NC; i += kThreads) {
            const uint32_t pt = a.grid[kGridIQ3S + i / NC];
            const __half2 lo = __floats2half2_rn((float) (2u * (pt & 7u) + 1u), (float) (2u * ((pt >> 3) & 7u) + 1u));
            const __half2 hi = __floats2half2_rn((float) (2u * ((pt >> 6) & 7u) + 1u), (float) (2u * ((pt >> 9) & 7u) + 1u));
            reinterpret_cast<uint2*>(lut)[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
        }
    }
    if (threadIdx.x < 4) zero[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);

    const int64_t n_rows = MODE == MODE_GU ? a.L.n_ff : a.L.n_embd;      // neurons (pairs) or down rows
    constexpr int kTileRows = MODE == MODE_GU ? 8 : 16;
    constexpr int kStepRows = kTiles * kTileRows;
    const int row_chunks = (n_gran + F::kGranules - 1) / F::kGranules;
    const int chunk0 = row_chunks * (warp % KS) / KS, n_chunks = row_chunks * (warp % KS + 1) / KS - chunk0;      // this warp's part of a row
    const int last_bytes = FMT == FMT_IQ1M ? (n_gran - 8 * (row_chunks - 1)) / 4 * 56       // bytes of a row in its last chunk
                         : FMT == FMT_IQ3S || PIECE == 16 ? kRowBytes : (n_gran - 4 * (row_chunks - 1)) * 36;
    const int pieces_per_col = (int) (K >> 3);               // 16-byte pieces of one image

    // this lane's copy duty inside a stage: pieces lane, lane + 32, ...; row = piece / kRowPieces
    // (IQ3_S: 55 words a row, a row at a time - lane and lane + 32 - so that no address lives in a register of its own)
    constexpr bool kByRow = FMT == FMT_IQ3S;
    constexpr int kRowPieces = kRowBytes / PIECE, kPieces = kRows * kRowPieces, kCopies = kByRow ? 1 : (kPieces + 31) / 32;
    int cp_row[kCopies], cp_off[kCopies];
    uint32_t cp_dst[kCopies];
#pragma unroll
    for (int j = 0; j < kCopies; ++j) {
        const int p = lane + 32 * j;
        cp_row[j] = p / kRowPieces;
        cp_off[j] = (p % kRowPieces) * PIECE;
        cp_dst[j] = (uint32_t) (cp_row[j] * kRowBytes + cp_off[j]);
    }

    pdl_wait();      // the table does not depend on earlier kernels; everything below does
    pdl_launch_dependents();
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
        if (work < work_end) next = items[item + 1];         // rides under this pass
        const int64_t r0 = (int64_t) rb * kStepRows + warp / KS * kTileRows;
        int live_tiles = 0;
        if (r0 < n_rows) live_tiles = (int) min((int64_t) steps, (n_rows - r0 + kStepRows - 1) / kStepRows);
        const int n_units = live_tiles * n_chunks;               // (tile, chunk) stages this warp streams for this part of the run
        const uint8_t* blob = reinterpret_cast<const uint8_t*>(pass.blob);
        const float* tail = reinterpret_cast<const float*>(blob + a.L.bytes - 16);
        // global address of this lane's pieces at chunk 0
        const uint8_t* src[kCopies];
#pragma unroll
        for (int j = 0; j < kCopies; ++j) {
            const int row = kByRow ? 0 : cp_row[j];
            const uint8_t* rp;
            if (MODE == MODE_GU)
                rp = row < 8 ? blob + (size_t) (r0 + row) * a.L.gu_row : blob + a.L.up_off + (size_t) (r0 + row - 8) * a.L.up_row;
            else
                rp = blob + a.L.down_off + (size_t) (r0 + row) * a.L.d_row;
            src[j] = rp + cp_off[j] + (size_t) chunk0 * kRowBytes;
        }
        // row 8's distance from row 0 (the first up row from the first gate row), and a row's from the one before it in each half
        const size_t row8 = MODE == MODE_GU ? (size_t) a.L.up_off + (size_t) r0 * (a.L.up_row - a.L.gu_row) : 8 * (size_t) a.L.d_row;
        const size_t pitch0 = MODE == MODE_GU ? (size_t) a.L.gu_row : (size_t) a.L.d_row, pitch1 = MODE == MODE_GU ? (size_t) a.L.up_row : (size_t) a.L.d_row;
        const size_t tile_bytes = (size_t) kStepRows * (MODE == MODE_GU ? a.L.gu_row : a.L.d_row);
        // the next (tile, chunk) unit to request and its global byte offset from the tile-0, chunk-0 addresses
        int iss_unit = 0, iss_chunk = 0;
        size_t iss_off = 0;
        auto issue = [&]() {
            if (iss_unit < n_units) {
                const uint32_t dst = wring_s + (uint32_t) (iss_unit % kStages) * kStageB;
                const int row_bytes = chunk0 + iss_chunk + 1 < row_chunks ? kRowBytes : last_bytes;
                if constexpr (kByRow) {
#pragma unroll
                    for (int row = 0; row < kRows; ++row) {
                        const uint8_t* p = src[0] + iss_off + (row < 8 ? row * pitch0 : row8 + (row - 8) * pitch1);
                        const uint32_t d = dst + (uint32_t) (row * kRowBytes + 4 * lane);
                        cp_async_piece<PIECE>(d, p);
                        if (lane < kRowPieces - 32) cp_async_piece<PIECE>(d + 128, p + 128);
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < kCopies; ++j)
                        if (lane + 32 * j < kPieces && (PIECE == 16 || cp_off[j] < row_bytes)) cp_async_piece<PIECE>(dst + cp_dst[j], src[j] + iss_off);
                }
                ++iss_unit;
                if (++iss_chunk == n_chunks) {
                    iss_chunk = 0;
                    iss_off += tile_bytes - (size_t) (n_chunks - 1) * kRowBytes;
                } else {
                    iss_off += kRowBytes;
                }
            }
            cp_async_commit();
        };
        {
            const int eb = pass.eb, ntok = pass.ntok;
            const int ncol = ntok * TERMS;
            __syncthreads();   // the previous pass is done with xs and s_ir
            if (threadIdx.x < ntok)
                s_ir[threadIdx.x] = (MODE == MODE_GU && a.n_x_rows > 0) ? a.ent_tok[eb + threadIdx.x] : eb + (int) threadIdx.x;
            __syncthreads();
            // the activation columns: image piece q of column c goes to piece ((q >> 2) * 8 + c) * 4 + (q & 3) of xs
            for (int i = threadIdx.x; i < ncol * pieces_per_col; i += kThreads) {
                const int c = i / pieces_per_col, q = i - c * pieces_per_col;
                const int ir = s_ir[c / TERMS], term = c % TERMS;
                const __half* sp = img + ((size_t) ir * TERMS + term) * K + (size_t) q * 8;
                cp_async16(xs_s + (uint32_t) ((((q >> 2) * kCols + c) * 4 + (q & 3)) * 16), sp);
            }
            cp_async_commit();
            // the weight stream
            iss_unit = 0;
            iss_chunk = 0;
            iss_off = 0;
#pragma unroll
            for (int c = 0; c < kStages - 1; ++c) issue();
            cp_async_wait<kStages - 1>();   // the activation group (the oldest) has landed
            __syncthreads();

            // per-pass epilogue constants, fetched before the stream starts so that no tile's epilogue waits on global memory:
            // the columns' inverse row scales times the tail scale(s) and the 2^8 of the fp16 block scales, and the output rows
            float f0 = 0.f, f1 = 0.f;
            int64_t o0 = 0, o1 = 0;
            {
                const int j0 = TERMS == 1 ? 2 * t : t, j1 = 2 * t + 1;
                if (j0 < ntok) f0 = inv[s_ir[j0]] * F::kUnscale;
                if (TERMS == 1 && j1 < ntok) f1 = inv[s_ir[j1]] * F::kUnscale;
                if (MODE == MODE_GU) {
                    o0 = (int64_t) (eb + j0) * a.L.n_ff;
                    o1 = (int64_t) (eb + j1) * a.L.n_ff;
                } else {
                    if (j0 < ntok) o0 = (int64_t) a.ent_dst[eb + j0] * a.L.n_embd;
                    if (TERMS == 1 && j1 < ntok) o1 = (int64_t) a.ent_dst[eb + j1] * a.L.n_embd;
                }
            }
            float sg = 1.f, su = 1.f, sd = 1.f;
            if constexpr (FMT == FMT_NVFP4) { sg = tail[0]; su = tail[1]; sd = tail[2]; }
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
            // this lane's B fragments: its column's pieces, or (column unused in this pass) the zero area with stride 0
            const bool col_live = g < ncol;
            const uint4* bcol = col_live ? reinterpret_cast<const uint4*>(xs) + g * 4 + t : zero;
            const int bstep = col_live ? 2 * kCols * 4 : 0;      // uint4 per 64-column granule
            const int bhalf = col_live ? kCols * 4 : 0;          // the second half-granule
            int tile = 0, chunk = 0;
            for (int unit = 0; unit < n_units; ++unit) {
                issue();
                cp_async_wait<kStages - 1>();
                __syncwarp();
                const uint8_t* st = wring + (size_t) (unit % kStages) * kStageB;
                const uint32_t* ra = reinterpret_cast<const uint32_t*>(st + g * kRowBytes);          // row g
                const uint32_t* rb = reinterpret_cast<const uint32_t*>(st + (g + 8) * kRowBytes);    // row g + 8
                const uint4* bp = bcol + (size_t) (chunk0 + chunk) * F::kGranules * bstep;
                if constexpr (FMT != FMT_NVFP4) {
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        if (FMT == FMT_IQ1M && 8 * (chunk0 + chunk) + 4 * b >= n_gran) break;       // past the row's last block
                        const uint8_t* ba = reinterpret_cast<const uint8_t*>(ra) + kRowBytes / 2 * b;
                        const uint8_t* bb = reinterpret_cast<const uint8_t*>(rb) + kRowBytes / 2 * b;
                        float sum[4] = {0.f, 0.f, 0.f, 0.f};
                        float da, db;
                        if constexpr (FMT == FMT_IQ1M) {
                            da = __half2float(__ushort_as_half((unsigned short) iq1m_d_bits(*reinterpret_cast<const uint2*>(ba + 48))));
                            db = __half2float(__ushort_as_half((unsigned short) iq1m_d_bits(*reinterpret_cast<const uint2*>(bb + 48))));
                        } else {
                            da = __half2float(*reinterpret_cast<const __half*>(ba));
                            db = __half2float(*reinterpret_cast<const __half*>(bb));
                        }
#pragma unroll
                        for (int gr = 0; gr < 4; ++gr) {
                            const uint4 b0 = bp[(4 * b + gr) * bstep], b1 = bp[(4 * b + gr) * bstep + bhalf];
                            uint32_t qa[8], qb[8];
                            if constexpr (FMT == FMT_IQ1M) {
                                // the sub-block's two index bytes, its byte of high bits, its 3 bits of the granule's scale word
                                auto units = [&](const uint8_t* blk, uint32_t (&q)[8]) {
                                    iq1m_units_16(*reinterpret_cast<const uint16_t*>(blk + 8 * gr + 2 * t), blk[32 + 4 * gr + t],
                                                  (*reinterpret_cast<const uint16_t*>(blk + 48 + 2 * gr) >> (3 * t)) & 7u, reinterpret_cast<const uint16_t*>(lut), q);
                                };
                                units(ba, qa);
                                units(bb, qb);
                            } else {
                                iq3s_16<NC>(ba, gr, t, reinterpret_cast<const uint2*>(lut) + (lane & (NC - 1)), qa);
                                iq3s_16<NC>(bb, gr, t, reinterpret_cast<const uint2*>(lut) + (lane & (NC - 1)), qb);
                            }
                            float s0[4], s1[4], s2[4], s3[4];
                            mma_f16_zero(s0, qa[0], qb[0], qa[1], qb[1], b0.x, b0.y);
                            mma_f16_zero(s1, qa[2], qb[2], qa[3], qb[3], b0.z, b0.w);
                            mma_f16_zero(s2, qa[4], qb[4], qa[5], qb[5], b1.x, b1.y);
                            mma_f16_zero(s3, qa[6], qb[6], qa[7], qb[7], b1.z, b1.w);
#pragma unroll
                            for (int i = 0; i < 4; ++i) sum[i] += (s0[i] + s1[i]) + (s2[i] + s3[i]);
                        }
#pragma unroll
                        for (int i = 0; i < 4; ++i) acc[i] = fmaf(sum[i], i < 2 ? da : db, acc[i]);
                    }
                } else {
                    float sum[4] = {0.f, 0.f, 0.f, 0.f};       // a chunk's sum, so that the row's is a short chain
#pragma unroll
                    for (int blk = 0; blk < 4; ++blk) {
                        if (PIECE != 16 && 4 * (chunk0 + chunk) + blk >= n_gran) break;   // past the row's last block
                        const uint4 b0 = bp[blk * bstep], b1 = bp[blk * bstep + bhalf];
                        const uint32_t sa = lut[reinterpret_cast<const uint8_t*>(ra)[36 * blk + t]];
                        const uint32_t sb = lut[reinterpret_cast<const uint8_t*>(rb)[36 * blk + t]];
                        uint32_t qa0[4], qa1[4], qb0[4], qb1[4];
                        cvt_e2m1x8(ra[9 * blk + 1 + 2 * t], qa0);
                        cvt_e2m1x8(ra[9 * blk + 2 + 2 * t], qa1);
                        cvt_e2m1x8(rb[9 * blk + 1 + 2 * t], qb0);
                        cvt_e2m1x8(rb[9 * blk + 2 + 2 * t], qb1);
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            qa0[i] = hmul2_bits(qa0[i], sa);
                            qa1[i] = hmul2_bits(qa1[i], sa);
                            qb0[i] = hmul2_bits(qb0[i], sb);
                            qb1[i] = hmul2_bits(qb1[i], sb);
                        }
                        float s0[4], s1[4], s2[4], s3[4];
                        mma_f16_zero(s0, qa0[0], qb0[0], qa0[1], qb0[1], b0.x, b0.y);
                        if constexpr (CHAIN == 1) {
                            mma_f16_zero(s1, qa0[2], qb0[2], qa0[3], qb0[3], b0.z, b0.w);
                            mma_f16_zero(s2, qa1[0], qb1[0], qa1[1], qb1[1], b1.x, b1.y);
                            mma_f16_zero(s3, qa1[2], qb1[2], qa1[3], qb1[3], b1.z, b1.w);
#pragma unroll
                            for (int i = 0; i < 4; ++i) sum[i] += (s0[i] + s1[i]) + (s2[i] + s3[i]);
                        } else {
                            mma_f16(s0, qa0[2], qb0[2], qa0[3], qb0[3], b0.z, b0.w);
                            mma_f16(s0, qa1[0], qb1[0], qa1[1], qb1[1], b1.x, b1.y);
                            mma_f16(s0, qa1[2], qb1[2], qa1[3], qb1[3], b1.z, b1.w);
#pragma unroll
                            for (int i = 0; i < 4; ++i) sum[i] += s0[i];
                        }
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[i] += sum[i];
                }
                __syncwarp();   // every lane is done with this stage before a later issue overwrites it
                if (++chunk != n_chunks) continue;
                // the tile is complete: undo the row scale and the 2^-8 of the fp16 block scales, apply the tail scales
                const int64_t rt = r0 + (int64_t) tile * kStepRows;
                chunk = 0;
                if constexpr (KS > 1) {
                    // the tile's other warps hand their sums to its first; two buffers, so one barrier of the tile's warps is enough: a
                    // buffer is written again only after the barrier of the tile in between, which its reader has passed
                    float4* buf = part + ((size_t) (tile & 1) * kTiles + warp / KS) * (KS - 1) * 32 + lane;
                    if (warp % KS != 0) buf[(warp % KS - 1) * 32] = make_float4(acc[0], acc[1], acc[2], acc[3]);
                    asm volatile("bar.sync %0, %1;\n" ::"r"(1 + warp / KS), "n"(KS * 32) : "memory");
                    if (warp % KS == 0)
#pragma unroll
                        for (int k = 0; k < KS - 1; ++k) {
                            const float4 o = buf[k * 32];
                            acc[0] += o.x; acc[1] += o.y; acc[2] += o.z; acc[3] += o.w;
                        }
                }
                ++tile;
                const float c0 = acc[0], c1 = acc[1], c2 = acc[2], c3 = acc[3];
                acc[0] = acc[1] = acc[2] = acc[3] = 0.f;
                if (KS > 1 && warp % KS != 0) continue;
                if (MODE == MODE_GU) {
                    if (TERMS == 1) {
                        if (2 * t < ntok) a.h[o0 + rt + g] = swiglu(c0 * f0 * sg, c2 * f0 * su, a.L);
                        if (2 * t + 1 < ntok) a.h[o1 + rt + g] = swiglu(c1 * f1 * sg, c3 * f1 * su, a.L);
                    } else if (t < ntok) {
                        a.h[o0 + rt + g] = swiglu((c0 + c1) * f0 * sg, (c2 + c3) * f0 * su, a.L);
                    }
                } else {
                    if (TERMS == 1) {
                        if (2 * t < ntok) {
                            store_out(a.out, a.out_kind, o0 + rt + g, c0 * f0 * sd);
                            store_out(a.out, a.out_kind, o0 + rt + g + 8, c2 * f0 * sd);
                        }
                        if (2 * t + 1 < ntok) {
                            store_out(a.out, a.out_kind, o1 + rt + g, c1 * f1 * sd);
                            store_out(a.out, a.out_kind, o1 + rt + g + 8, c3 * f1 * sd);
                        }
                    } else if (t < ntok) {
                        store_out(a.out, a.out_kind, o0 + rt + g, (c0 + c1) * f0 * sd);
                        store_out(a.out, a.out_kind, o0 + rt + g + 8, (c2 + c3) * f0 * sd);
                    }
                }
            }
            cp_async_wait<0>();
        }
    }
    cp_async_wait<0>();
}

// shared memory that a block may ask for, alone on its SM or one of two (227 and 113 KB less the static words)
constexpr size_t kSmemOne = 232448 - 256, kSmemTwo = 115712 - 256;

template <int FMT>
size_t smem_bytes(int64_t K, int W, int ST, int NC, int KS) {
    return (size_t) K * kCols * 2 + (size_t) Fmt<FMT>::kTable * NC + 128 + (size_t) W * ST * kStageBytes<FMT> + (size_t) 2 * (W / KS) * (KS - 1) * 512;
}
// the widest rows: those whose columns leave room for a ring (what this kernel has taken from the start)
template <int FMT>
bool fits(int64_t K) { return (size_t) K * kCols * 2 + Fmt<FMT>::kTable + 128 + 32 * kStageBytes<FMT> <= 200 * 1024; }
size_t align256(size_t v) { return (v + 255) & ~(size_t) 255; }

template <int FMT, int MODE, int TERMS, int PIECE, int CHAIN, int W, int OCC, int ST, int NC, int KS>
int32_t launch_as(const ExpertArgs& a, const __half* img, const float* inv, const PassRec* items, const int* n_items, cudaStream_t st) {
    const size_t smem = smem_bytes<FMT>(MODE == MODE_GU ? a.L.n_embd : a.L.n_ff, W, ST, NC, KS);
    static std::atomic<bool> configured[64];   // per device; threads of different devices call concurrently
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return (int32_t) cudaErrorInvalidDevice;
    if (!configured[dev].load(std::memory_order_acquire)) {
        const cudaError_t e = cudaFuncSetAttribute(blk_mma_kernel<FMT, MODE, TERMS, PIECE, CHAIN, W, OCC, ST, NC, KS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   (int) (OCC == 2 ? kSmemTwo : kSmemOne));
        if (e != cudaSuccess) return (int32_t) e;
        configured[dev].store(true, std::memory_order_release);
    }
    const int64_t rows = MODE == MODE_GU ? a.L.n_ff : a.L.n_embd, step_rows = (MODE == MODE_GU ? 8 : 16) * (W / KS);
    launch_k(blk_mma_kernel<FMT, MODE, TERMS, PIECE, CHAIN, W, OCC, ST, NC, KS>, dim3((unsigned) (OCC * sm_count())), dim3(W * 32), smem, st, a, img, inv, items, n_items,
             (int) ((rows + step_rows - 1) / step_rows));
    return launch_status();
}

// Sixteen warps an SM either way: two blocks of eight where shared memory holds two, which hide each other's first loads, else one of
// sixteen.  (Four stages a warp left one block of eight: 2560-column NVFP4 rows and every IQ3_S row.)  IQ3_S is bound by its look-ups,
// eight bytes at 32 unrelated points: sixteen copies of the codebook, a lane's own in two banks of its own, take the bank conflicts away
// (4 passes over the banks a look-up on average without them), which one block of sixteen warps has room for.
template <int FMT, int MODE, int TERMS, int PIECE, int CHAIN>
int32_t launch(const ExpertArgs& a, const __half* img, const float* inv, const PassRec* items, const int* n_items, cudaStream_t st) {
    const int64_t K = MODE == MODE_GU ? a.L.n_embd : a.L.n_ff, rows = MODE == MODE_GU ? a.L.n_ff : a.L.n_embd;
    const bool two = FMT != FMT_IQ3S && smem_bytes<FMT>(K, 8, 3, 1, 4) <= kSmemTwo;
    const bool copies = FMT == FMT_IQ3S && smem_bytes<FMT>(K, 16, 2, 16, 4) <= kSmemOne;
    // columns are split where whole rows would leave a block few steps, so that the last, partial one weighs little: IQ3_S up to eight
    // steps (24 tokens of 2048 x 512, 512 experts, 7.4 steps: 202 us whole, 193 split in two), NVFP4, whose decode costs less beside the
    // sums' exchange, up to four (16 tokens of 2560 x 640, 6.2 steps: 123 whole, 130 split).  cap_groups and cap_entries bound the passes
    // on the host
    const int64_t chunks = FMT == FMT_NVFP4 ? (K + 255) / 256 : (K + 511) / 512, step_rows = (MODE == MODE_GU ? 8 : 16) * (two ? 8 : 16);
    const int64_t steps = (a.cap_groups + a.cap_entries / (kCols / TERMS)) * ((rows + step_rows - 1) / step_rows);
    int ks = 1;
    while (ks < 4 && chunks >= 2 * ks && steps * ks < (FMT == FMT_NVFP4 ? 4 : 8) * (int64_t) sm_count() * (two ? 2 : 1)) ks *= 2;
#define BLK_AS(W, OCC, ST, NC) \
    do { \
        if (ks == 4) return launch_as<FMT, MODE, TERMS, PIECE, CHAIN, W, OCC, ST, NC, 4>(a, img, inv, items, n_items, st); \
        if (ks == 2) return launch_as<FMT, MODE, TERMS, PIECE, CHAIN, W, OCC, ST, NC, 2>(a, img, inv, items, n_items, st); \
        return launch_as<FMT, MODE, TERMS, PIECE, CHAIN, W, OCC, ST, NC, 1>(a, img, inv, items, n_items, st); \
    } while (0)
    if constexpr (FMT != FMT_IQ3S) {
        if (two) BLK_AS(8, 2, 3, 1);
    } else {
        if (copies) BLK_AS(16, 1, 2, 16);
    }
    BLK_AS(16, 1, 2, 1);
#undef BLK_AS
}

}  // namespace

// scratch beyond the SwiGLU buffer: the x images (up to two fp16 terms), the h images (two terms), the inverse row scales
size_t experts_mma_scratch_bytes(int64_t cap_entries, int64_t n_embd, int64_t n_ff) {
    // the pass list: at most one pass per entry, 16 bytes each, plus its count
    return align256((size_t) cap_entries * n_embd * 4) + align256((size_t) cap_entries * n_ff * 4) + 2 * align256((size_t) cap_entries * 4) +
           align256((size_t) (cap_entries + 1) * 16 + 16);
}

int32_t experts_grouped_mma(const ExpertArgs& a, bool iq1m, cudaStream_t st) {
    const bsx_expert_layout& L = a.L;
    // NVFP4: gate and up rows are whole 256-column chunks (n_embd % 256 == 0 in every layout), down rows whole 64-column blocks.
    // IQ3_S: rows of whole 512-column chunks (every other 110-byte block starts on 4 bytes, what the copies need).  IQ1_M: whole blocks of
    // 256 columns.  The activation image must fit shared memory.
    const int fmt = L.gu_type == kTypeNVFP4 ? FMT_NVFP4 : L.gu_type == kTypeIQ3S ? FMT_IQ3S : FMT_IQ1M;
    const bool whole = L.n_ff % 256 == 0;
    if ((L.gu_type != kTypeNVFP4 && L.gu_type != kTypeIQ3S && !(iq1m && L.gu_type == kTypeIQ1M)) || L.up_type != L.gu_type || L.d_type != L.gu_type) return BSX_E_TYPE;
    if (fmt == FMT_NVFP4) {
        if (L.n_embd % 256 || L.n_ff % 64) return BSX_E_TYPE;
        if (!fits<FMT_NVFP4>(L.n_embd) || !fits<FMT_NVFP4>(L.n_ff)) return BSX_E_TYPE;
    } else if (fmt == FMT_IQ3S) {
        if (L.n_embd % 512 || L.n_ff % 512) return BSX_E_TYPE;
        if (!fits<FMT_IQ3S>(L.n_embd) || !fits<FMT_IQ3S>(L.n_ff)) return BSX_E_TYPE;
    } else {
        if (L.n_embd % 256 || L.n_ff % 256) return BSX_E_TYPE;
        if (!fits<FMT_IQ1M>(L.n_embd) || !fits<FMT_IQ1M>(L.n_ff)) return BSX_E_TYPE;
    }
    // scratch: [h fp32][x images][h images][x inverse scales][h inverse scales]
    uint8_t* p = reinterpret_cast<uint8_t*>(a.h) + align256((size_t) a.cap_entries * L.n_ff * 4);
    __half* ximg = reinterpret_cast<__half*>(p);
    p += align256((size_t) a.cap_entries * L.n_embd * 4);
    __half* himg = reinterpret_cast<__half*>(p);
    p += align256((size_t) a.cap_entries * L.n_ff * 4);
    float* xinv = reinterpret_cast<float*>(p);
    float* hinv = xinv + align256((size_t) a.cap_entries * 4) / 4;
    int* n_items = reinterpret_cast<int*>(hinv + align256((size_t) a.cap_entries * 4) / 4);
    PassRec* items = reinterpret_cast<PassRec*>(n_items + 4);
    const int phase = experts_phase(a.L);
    // a warp per image row, 8 a block, plus the block that lists the passes
    const int64_t x_rows = a.n_x_rows > 0 ? a.n_x_rows : a.cap_entries;
    const unsigned nbx = (unsigned) ((x_rows + 7) / 8 + 1), nbh = (unsigned) ((a.cap_entries + 7) / 8 + 1);
    int32_t rc = BSX_OK;
    if (phase != 2) {
        if (a.x_kind == BSX_X_BF16) {
            launch_k(fmt == FMT_IQ3S ? prep_image_kernel<FMT_IQ3S, false, 1> : prep_image_kernel<FMT_NVFP4, false, 1>, dim3(nbx), dim3(256), 0, st, a, ximg, xinv, items, n_items);
            rc = fmt == FMT_IQ3S ? launch<FMT_IQ3S, MODE_GU, 1, 4, 1>(a, ximg, xinv, items, n_items, st)
                 : fmt == FMT_IQ1M ? launch<FMT_IQ1M, MODE_GU, 1, 8, 1>(a, ximg, xinv, items, n_items, st)
                 : whole         ? launch<FMT_NVFP4, MODE_GU, 1, 16, 4>(a, ximg, xinv, items, n_items, st)
                                 : launch<FMT_NVFP4, MODE_GU, 1, 16, 1>(a, ximg, xinv, items, n_items, st);
        } else {
            launch_k(fmt == FMT_IQ3S ? prep_image_kernel<FMT_IQ3S, false, 2> : prep_image_kernel<FMT_NVFP4, false, 2>, dim3(nbx), dim3(256), 0, st, a, ximg, xinv, items, n_items);
            rc = fmt == FMT_IQ3S ? launch<FMT_IQ3S, MODE_GU, 2, 4, 1>(a, ximg, xinv, items, n_items, st)
                 : fmt == FMT_IQ1M ? launch<FMT_IQ1M, MODE_GU, 2, 8, 1>(a, ximg, xinv, items, n_items, st)
                 : whole         ? launch<FMT_NVFP4, MODE_GU, 2, 16, 4>(a, ximg, xinv, items, n_items, st)
                                 : launch<FMT_NVFP4, MODE_GU, 2, 16, 1>(a, ximg, xinv, items, n_items, st);
        }
    }
    if (rc != BSX_OK || phase == 1) return rc;
    rc = fmt == FMT_IQ3S ? launch_spread<prep_image_kernel<FMT_IQ3S, true, 2>>(nbh, st, a, himg, hinv, items, n_items)
                         : launch_spread<prep_image_kernel<FMT_NVFP4, true, 2>>(nbh, st, a, himg, hinv, items, n_items);
    if (rc != BSX_OK) return rc;
    if (fmt == FMT_IQ3S) return launch<FMT_IQ3S, MODE_DOWN, 2, 4, 1>(a, himg, hinv, items, n_items, st);
    if (fmt == FMT_IQ1M) return launch<FMT_IQ1M, MODE_DOWN, 2, 8, 1>(a, himg, hinv, items, n_items, st);
    // Down rows of n_ff columns: the copies' width is what their start is aligned to.  An n_ff that is not whole 256-column chunks
    // went to the warp-per-row kernels before (2 % of the copy bandwidth: fp32 decode and FMA for every weight and entry); here
    // the same 27-token step (2560 x 640, 512 + 1 experts, top-10) takes 170 us instead of 3648.
    if (whole) return launch<FMT_NVFP4, MODE_DOWN, 2, 16, 4>(a, himg, hinv, items, n_items, st);
    if (L.n_ff % 128 == 0) return launch<FMT_NVFP4, MODE_DOWN, 2, 8, 1>(a, himg, hinv, items, n_items, st);
    return launch<FMT_NVFP4, MODE_DOWN, 2, 4, 1>(a, himg, hinv, items, n_items, st);
}

}  // namespace bsx
