// router_softmax.cuh - the one-warp-per-token fp32 softmax top-k router, included by two translation units: router.cu
// (IEEE expf and division; the Basalt prompt path's route_kernel, src/models/qwen4exp/prefill/kernels.cu:351-390) and
// router_fast.cu (built with --use_fast_math, weight = p * (1 / sum); the decode path's route,
// src/models/qwen4exp/kernels/native_router.cu:44-99).  The including file defines BSX_SOFTMAX_KERNEL (the kernel's name)
// BSX_SOFTMAX_TOKEN (the per-token device routine's name) and BSX_SOFTMAX_RECIPROCAL (0: divide, 1: multiply by the reciprocal).
//
// Arithmetic order, which fixes every bit of the result: lane l holds experts l, l+32, ...; max over all experts; per lane
// v = expf(v - max) summed in index order, lanes summed by xor butterfly; v *= 1/sum; NaN -> -FLT_MAX; k argmax passes
// (value descending, index ascending); the chosen probabilities are added per WINNING lane in selection order, lanes summed
// by butterfly, clamped below at 2^-14.  The reference instantiates 512 and 256 experts with k = 10 only; this is the same
// sequence for any E % 32 == 0 (E <= 1024) and k <= 32.
#include <cfloat>

#include "common.cuh"
#include "pdl.cuh"

namespace bsx {

// one token by one warp: lg = the token's E logits; ids / wout = its k outputs; keys: 33 REGT words of the warp's own (unused for REGT = 0).
// Returns the id of rank `lane` (lane < k).
template <int REGT>
__device__ __forceinline__ int BSX_SOFTMAX_TOKEN(const float* lg, int32_t* __restrict__ ids, float* __restrict__ wout, int E, int k, uint32_t* keys) {
    constexpr int MAXR = REGT > 0 ? REGT : 32;
    const int lane = threadIdx.x & 31;
    const int reg = REGT > 0 ? REGT : (E >> 5);
    float v[MAXR];
#pragma unroll
    for (int i = 0; i < MAXR; ++i) v[i] = i < reg ? lg[lane + i * 32] : -INFINITY;
    float mx = -INFINITY;
#pragma unroll
    for (int i = 0; i < MAXR; ++i)
        if (i < reg) mx = fmaxf(mx, v[i]);
    mx = warp_max_xor(mx);
    float sum = 0.0f;
#pragma unroll
    for (int i = 0; i < MAXR; ++i)
        if (i < reg) { v[i] = expf(v[i] - mx); sum += v[i]; }
    const float rcp = 1.0f / warp_sum_xor(sum);
#pragma unroll
    for (int i = 0; i < MAXR; ++i)
        if (i < reg) { v[i] *= rcp; if (isnan(v[i])) v[i] = -FLT_MAX; }
    // k argmax passes (value descending, index ascending).  Floats are compared through an order-preserving map to
    // unsigned integers, so the warp-wide maximum and the lowest index holding it are one redux instruction each; a lane
    // keeps the maximum of its own values and only the winning lane rescans.  (+0 and -0 would order differently from the
    // float compare, but a probability here is +0 at the lowest, and the markers -FLT_MAX and -inf are distinct values.)
    // The values stay in registers: every index into v[] below is a compile-time constant.  (Reading "the winner's value" as
    // v[ex >> 5] makes the compiler put the array in local memory, and the selection becomes a chain of L1 round trips -
    // measured ~6 us a token.)  A chosen value is recovered from its key, and chosen positions are remembered in a bit mask.
    float selected = 0.0f, selected_sum = 0.0f;
    auto key = [](float f) { const uint32_t b = __float_as_uint(f); return (b & 0x80000000u) ? ~b : (b | 0x80000000u); };
    auto unkey = [](uint32_t q) { return __uint_as_float((q & 0x80000000u) ? (q & 0x7FFFFFFFu) : ~q); };
    uint32_t kv[MAXR];
#pragma unroll
    for (int i = 0; i < MAXR; ++i) kv[i] = i < reg ? key(v[i]) : 0u;
    uint32_t lmax = 0u, taken = 0u;
    int lidx = 0;
    auto rescan = [&]() {
        lmax = 0u;       // below every key (the key of -inf is 0x007FFFFF)
        lidx = 0;
#pragma unroll
        for (int i = 0; i < MAXR; ++i)
            if (i < reg && !((taken >> i) & 1u) && kv[i] > lmax) { lmax = kv[i]; lidx = i; }
    };
    rescan();
    int my_id = 0;
    if constexpr (REGT > 0) {
        // A rank is a chain of dependent steps, so the rescan of the winning lane's values (64 instructions with one lane active) is
        // shared out: value i of every lane also lies in row i of `keys`, which lane i alone reads and writes.
        // Selection + plan of one token, 512 experts, top 10, after the logits: 5.1 us -> 4.3; of 8 tokens 8.2 -> 6.6 (with the ids kept in
        // registers instead of read back).
#pragma unroll
        for (int i = 0; i < REGT; ++i) keys[i * 33 + lane] = kv[i];
        __syncwarp();
        for (int rank = 0; rank < k; ++rank) {
            const uint32_t gmax = __reduce_max_sync(kFull, lmax);
            const int ex = (int) __reduce_min_sync(kFull, lmax == gmax ? (unsigned) (lane + lidx * 32) : 0xFFFFFFFFu);
            const int wl = ex & 31;
            uint32_t q = 0u;
            if (lane < REGT) {
                q = keys[lane * 33 + wl];
                if (lane == (ex >> 5)) keys[lane * 33 + wl] = q = 0u;
            }
            const uint32_t next = __reduce_max_sync(kFull, q);
            const int at = __ffs(__ballot_sync(kFull, q == next)) - 1;      // the lowest index holding it (0 when none is left: never chosen)
            const float best = unkey(gmax);
            if (wl == lane) {
                selected_sum += best;
                lmax = next;
                lidx = at;
            }
            if (rank == lane) {
                selected = best;
                my_id = ex;
            }
        }
    } else {
        for (int rank = 0; rank < k; ++rank) {
            const uint32_t gmax = __reduce_max_sync(kFull, lmax);
            const int ex = (int) __reduce_min_sync(kFull, lmax == gmax ? (unsigned) (lane + lidx * 32) : 0xFFFFFFFFu);
            const float best = unkey(gmax);
            if ((ex & 31) == lane) {
                taken |= 1u << lidx;
                selected_sum += best;
                rescan();
            }
            if (rank == lane) {
                selected = best;
                my_id = ex;
            }
        }
    }
    if (lane < k) ids[lane] = my_id;
    selected_sum = fmaxf(warp_sum_xor(selected_sum), 6.103515625e-5f);
#if BSX_SOFTMAX_RECIPROCAL
    const float inv = 1.0f / selected_sum;
    if (lane < k) wout[lane] = selected * inv;
#else
    if (lane < k) wout[lane] = selected / selected_sum;
#endif
    return my_id;
}

template <int REGT>
__global__ void __launch_bounds__(256) BSX_SOFTMAX_KERNEL(const float* logits, int32_t* __restrict__ ids,
                                                         float* __restrict__ wout, int64_t T, int E, int k) {
    __shared__ uint32_t keys[8][REGT > 0 ? REGT * 33 : 1];
    pdl_wait();
    pdl_launch_dependents();
    const int64_t t = (int64_t) blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (t >= T) return;
    BSX_SOFTMAX_TOKEN<REGT>(logits + t * E, ids + t * k, wout + t * k, E, k, keys[threadIdx.x >> 5]);
}

static inline int32_t BSX_SOFTMAX_LAUNCH(const float* logits, int64_t T, int E, int k, int32_t* ids, float* w, cudaStream_t st) {
    // decode windows: two tokens a block, so the window's selections spread over the SMs instead of queueing on a few
    const unsigned wpb = T <= 256 ? 2u : 8u, blocks = (unsigned) ((T + wpb - 1) / wpb);
    switch (E >> 5) {
        case 2: launch_k(BSX_SOFTMAX_KERNEL<2>, dim3(blocks), dim3(32 * wpb), 0, st, logits, ids, w, T, E, k); break;
        case 4: launch_k(BSX_SOFTMAX_KERNEL<4>, dim3(blocks), dim3(32 * wpb), 0, st, logits, ids, w, T, E, k); break;
        case 8: launch_k(BSX_SOFTMAX_KERNEL<8>, dim3(blocks), dim3(32 * wpb), 0, st, logits, ids, w, T, E, k); break;
        case 12: launch_k(BSX_SOFTMAX_KERNEL<12>, dim3(blocks), dim3(32 * wpb), 0, st, logits, ids, w, T, E, k); break;
        case 16: launch_k(BSX_SOFTMAX_KERNEL<16>, dim3(blocks), dim3(32 * wpb), 0, st, logits, ids, w, T, E, k); break;
        default: launch_k(BSX_SOFTMAX_KERNEL<0>, dim3(blocks), dim3(32 * wpb), 0, st, logits, ids, w, T, E, k); break;
    }
    return launch_status();
}

}  // namespace bsx
