// fp16_rows.cuh - activation (and gate) rows as fp16 operand images, for the fp16 tensor-core kernels of prompt-sized batches.
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"
#include "experts.cuh"
#include "tc5.cuh"

namespace bsx {
namespace {

// rows [R][H] (fp32 or bf16) -> `terms` fp16 planes [terms][R][H], each row scaled by a power of two so its largest magnitude
// lands in [2^13, 2^14), k-permuted inside 16-column groups; inv[r] undoes the scale.  Plane 1 holds the rounding residual
// of plane 0.
struct PlaneRows {
    const void* x;
    int kind, terms;
    int64_t R;
    __half* img;
    float* inv;
};

// The rows of both operands in one launch: TPR threads a row, each with up to two of its 16-column groups in registers (a row is read
// once up to 32 TPR columns) and stored as two 16-byte pieces.  Bound by HBM.  With a warp a row, single values loaded and stored and a
// launch for each operand, 8192 bf16 rows of 7168 columns and 256 gate rows took 94 + 42 us and 777 fp32 rows of 5120 columns and 384 gate
// rows 28 + 26; the single plane of the prompt experts, 4096 bf16 rows of 7168 columns: 64 -> 27.
template <int TPR>
__global__ void __launch_bounds__(256) rows_to_fp16_planes_kernel(PlaneRows x, PlaneRows gate, int64_t H) {
    constexpr int kRows = 256 / TPR, kKeep = 2;
    __shared__ float s_max[8];
    const unsigned x_blocks = (unsigned) ((x.R + kRows - 1) / kRows);
    const bool is_x = blockIdx.x < x_blocks;
    const PlaneRows& a = is_x ? x : gate;
    const int64_t r = (int64_t) (is_x ? blockIdx.x : blockIdx.x - x_blocks) * kRows + threadIdx.x / TPR;
    const int tr = threadIdx.x % TPR, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool live = r < a.R;
    const int n_sb = live ? (int) (H >> 4) : 0;
    float v[kKeep][16];
    float amax = 0.f;
#pragma unroll
    for (int i = 0; i < kKeep; ++i) {
        if (tr + i * TPR < n_sb) {
            load16(a.x, a.kind, r, H, tr + i * TPR, v[i]);
#pragma unroll
            for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(v[i][j]));
        }
    }
    for (int sb = tr + kKeep * TPR; sb < n_sb; sb += TPR) {
        float w[16];
        load16(a.x, a.kind, r, H, sb, w);
#pragma unroll
        for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(w[j]));
    }
    amax = warp_max_xor(amax);
    if (lane == 0) s_max[warp] = amax;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TPR / 32; ++i) amax = fmaxf(amax, s_max[warp / (TPR / 32) * (TPR / 32) + i]);
    int ex = 0;
    float s = 1.f, iv = 1.f;
    if (amax > 0.f && amax <= 3.0e38f) {
        frexpf(amax, &ex);
        ex = max(-100, min(100, 14 - ex));
        s = ldexpf(1.f, ex);
        iv = ldexpf(1.f, -ex);
    }
    if (live && tr == 0) a.inv[r] = iv;
    auto store = [&](int sb, const float (&w)[16]) {
        uint32_t hi[8], lo[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {       // positions 2 i and 2 i + 1 of the permuted order: columns i and i + 8
            const float p = w[i] * s, q = w[i + 8] * s;
            const __half hp = __float2half_rn(p), hq = __float2half_rn(q);
            hi[i] = (uint32_t) __half_as_ushort(hp) | ((uint32_t) __half_as_ushort(hq) << 16);
            lo[i] = (uint32_t) __half_as_ushort(__float2half_rn(p - __half2float(hp))) | ((uint32_t) __half_as_ushort(__float2half_rn(q - __half2float(hq))) << 16);
        }
        uint4* o = reinterpret_cast<uint4*>(a.img + r * H + 16 * sb);
        o[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        o[1] = make_uint4(hi[4], hi[5], hi[6], hi[7]);
        if (a.terms > 1) {
            o = reinterpret_cast<uint4*>(a.img + (a.R + r) * H + 16 * sb);
            o[0] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
            o[1] = make_uint4(lo[4], lo[5], lo[6], lo[7]);
        }
    };
#pragma unroll
    for (int i = 0; i < kKeep; ++i)
        if (tr + i * TPR < n_sb) store(tr + i * TPR, v[i]);
    for (int sb = tr + kKeep * TPR; sb < n_sb; sb += TPR) {
        float w[16];
        load16(a.x, a.kind, r, H, sb, w);
        store(sb, w);
    }
}

}  // namespace
}  // namespace bsx
