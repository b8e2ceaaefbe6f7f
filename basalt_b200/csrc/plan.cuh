// plan.cuh - the decode-window plan as block-wide device routines, shared by the plan kernel (dispatch.cu) and the fused
// selection + plan kernel (router.cu).
//
// The plan (Basalt: moe_plan, src/models/inkling2/kernels/ops.cu:275-340): the experts that have pairs and a non-zero blob address
// become groups in ascending expert order; an expert's entries keep the order of the pairs (a pair's place = the number of
// earlier pairs naming the same expert, the reference's rule, ops.cu:331-339), so no position comes from an atomic.
//
// The step is latency, not work: one block, and everything it needs in shared memory.  Each expert has a count and a 64-bit mask of
// the tokens that name it, so a window of up to 64 tokens reads a pair's place off as the population count of the mask below the
// pair's token - no loop over the earlier pairs (which a token naming an expert twice, or more than 64 tokens, falls back to).  One
// block scan over the experts carries entries, groups and passes together in the fields of a 64-bit word.  Measured on a B200
// with 512 experts, top-10: the plan kernel of a 64-token window 8.1 us -> 4.1 after the selection before it, with the loop and three scans replaced; selection +
// plan of an 8-token window 11.2 -> 9.2, of one token 6.1 -> 5.1 (that kernel counted over all pairs of the window instead).
#pragma once
#include "common.cuh"

namespace bsx {

// a pass of the packed expert kernels: up to kPassEntries consecutive entries [eb, eb + ntok) of one group, with the group's blob
constexpr int kPassEntries = 8;
struct __align__(16) PassRec {
    unsigned long long blob;
    int eb, ntok;
};

// block-wide exclusive sum (blockDim a multiple of 32, at most 1024); *total = the block's sum; sh: 32 words
template <typename T>
__device__ inline T block_excl_sum(T v, T* total, T* sh) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    T x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const T y = __shfl_up_sync(kFull, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) sh[w] = x;
    __syncthreads();
    if (w == 0) {
        T s = lane < nw ? sh[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const T y = __shfl_up_sync(kFull, s, o);
            if (lane >= o) s += y;
        }
        sh[lane] = s;
    }
    __syncthreads();
    const T r = x - v + (w > 0 ? sh[w - 1] : 0);
    *total = sh[nw - 1];
    __syncthreads();
    return r;
}

struct PlanSmem {
    unsigned long long* blob;   // [E]
    unsigned long long* mask;   // [E]: the tokens naming the expert, or null (more than 64 tokens, no room, or places from a cursor)
    int32_t* count;             // [E]
    int32_t* first;             // [E]: the expert's first entry
    int32_t* twice;             // a token named one expert twice: the masks do not give places
    int32_t* sid;               // [n]: the pairs' ids (-1: no entry)
};
// A launch without an opt-in has 48 KB of shared memory in all, static (the scan's words in plan_finish) and dynamic together.
constexpr size_t kPlanSmemStatic = 32 * sizeof(unsigned long long);
constexpr size_t kPlanSmemMax = 48 * 1024 - kPlanSmemStatic;
constexpr int kPlanMaskTokens = 64;
__host__ __device__ inline size_t plan_smem_bytes(int E, int n, bool masks) { return (size_t) E * (masks ? 24 : 16) + 8 + (size_t) n * 4; }
// whether a window of n_tok tokens gets masks
__host__ __device__ inline bool plan_masks(int E, int n, int n_tok) { return n_tok <= kPlanMaskTokens && plan_smem_bytes(E, n, true) <= kPlanSmemMax; }
__device__ inline PlanSmem plan_smem(void* base, int E, bool masks) {
    PlanSmem s;
    s.blob = static_cast<unsigned long long*>(base);
    s.mask = masks ? s.blob + E : nullptr;
    s.count = reinterpret_cast<int32_t*>(s.blob + (masks ? 2 : 1) * E);
    s.first = s.count + E;
    s.twice = s.first + E;
    s.sid = s.twice + 2;
    return s;
}
// every thread of the block; a block barrier must follow before plan_note_pair
__device__ inline void plan_load_blobs(const PlanSmem& s, const unsigned long long* __restrict__ blobs, int E) {
    for (int e = threadIdx.x; e < E; e += blockDim.x) {
        s.blob[e] = blobs[e];
        s.count[e] = 0;
        if (s.mask) s.mask[e] = 0ull;
    }
    if (threadIdx.x == 0) *s.twice = 0;
}
// pair i of token t names expert e (any thread, once per pair); a block barrier must follow before plan_finish
__device__ inline void plan_note_pair(const PlanSmem& s, int i, int t, int e, int E) {
    if ((unsigned) e >= (unsigned) E || !s.blob[e]) e = -1;
    s.sid[i] = e;
    if (e < 0) return;
    atomicAdd(&s.count[e], 1);
    if (s.mask) {
        const unsigned long long bit = 1ull << t;
        if (atomicOr(&s.mask[e], bit) & bit) *s.twice = 1;
    }
}
// every thread of the block.  items / n_items (optional): the pass list of the packed expert kernels, made here so that no
// kernel of its own has to.  tok_base: the first token of the shared expert's group (its entries read tokens tok_base ..
// tok_base + n_tok - 1).  STABLE = false: an expert's entries take their places from a shared-memory cursor instead of by counting
// earlier pairs - for callers to whom the order of the entries inside a group does not matter (every entry writes its own row).
template <bool STABLE = true>
__device__ inline void plan_finish(const PlanSmem& s, int n, int k, int E, unsigned long long shared_blob, int n_tok,
                                   unsigned long long* __restrict__ ptr, int32_t* __restrict__ start, int32_t* __restrict__ n_groups,
                                   int32_t* __restrict__ dst, int32_t* __restrict__ tok, PassRec* __restrict__ items, int* __restrict__ n_items,
                                   int tok_base = 0) {
    __shared__ unsigned long long sh[kPlanSmemStatic / sizeof(unsigned long long)];
    constexpr int kField = 20;                                // entries | groups << 20 | passes << 40: none reaches 2^20 here
    constexpr unsigned long long kLow = (1ull << kField) - 1;
    int at = 0, g = 0, np_total = 0;   // running totals over the expert chunks of blockDim.x
    for (int e0 = 0; e0 < E; e0 += blockDim.x) {
        const int e = e0 + threadIdx.x;
        const int c = e < E ? s.count[e] : 0;
        const int np = (c + kPassEntries - 1) / kPassEntries;
        unsigned long long total = 0;
        const unsigned long long o = block_excl_sum<unsigned long long>(
            (unsigned long long) c | ((unsigned long long) (c > 0) << kField) | ((unsigned long long) np << (2 * kField)), &total, sh);
        const int first = at + (int) (o & kLow), grp = g + (int) ((o >> kField) & kLow), pass = np_total + (int) (o >> (2 * kField));
        if (e < E) s.first[e] = first;
        if (c > 0) {
            ptr[grp] = s.blob[e];
            start[grp] = first;
            if (items)
                for (int p = 0; p < np; ++p) {
                    PassRec r;
                    r.blob = s.blob[e];
                    r.eb = first + p * kPassEntries;
                    r.ntok = min(kPassEntries, c - p * kPassEntries);
                    items[pass + p] = r;
                }
        }
        at += (int) (total & kLow);
        g += (int) ((total >> kField) & kLow);
        np_total += (int) (total >> (2 * kField));
    }
    if (shared_blob != 0ull && n_tok > 0) {
        // the shared expert: one more group holding every token, its rows after the routed pairs' rows
        if (threadIdx.x == 0) {
            ptr[g] = shared_blob;
            start[g] = at;
        }
        for (int t = threadIdx.x; t < n_tok; t += blockDim.x) {
            dst[at + t] = n + t;
            tok[at + t] = tok_base + t;
        }
        if (items) {
            const int np = (n_tok + kPassEntries - 1) / kPassEntries;
            for (int p = threadIdx.x; p < np; p += blockDim.x) {
                PassRec r;
                r.blob = shared_blob;
                r.eb = at + p * kPassEntries;
                r.ntok = min(kPassEntries, n_tok - p * kPassEntries);
                items[np_total + p] = r;
            }
            np_total += np;
        }
        at += n_tok;
        ++g;
    }
    if (threadIdx.x == 0) {
        start[g] = at;
        start[g + 1] = at;
        *n_groups = g;
        if (n_items) n_items[0] = np_total;
    }
    __syncthreads();   // first[] is complete
    const bool by_mask = STABLE && s.mask && *s.twice == 0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int e = s.sid[i];
        if (e < 0) continue;
        const int t = i / k;
        int p;
        if (by_mask) {
            p = s.first[e] + __popcll(s.mask[e] & ((1ull << t) - 1ull));
        } else if (STABLE) {
            int before = 0;
            int j = 0;
            for (; j + 4 <= i; j += 4) before += (s.sid[j] == e) + (s.sid[j + 1] == e) + (s.sid[j + 2] == e) + (s.sid[j + 3] == e);
            for (; j < i; ++j) before += s.sid[j] == e;
            p = s.first[e] + before;
        } else {
            p = atomicAdd(&s.first[e], 1);
        }
        dst[p] = i;
        tok[p] = t;
    }
}

}  // namespace bsx
