// experts_prefill.cu - prompt-sized grouped experts for NVFP4 blobs on the 5th-generation tensor cores (tcgen05).
//
// A ragged grouped GEMM over the dispatch's expert-sorted rows: for every 128-row tile of one expert,
//   gate/up:  [128 rows x H] . [H x 2I]  -> SwiGLU ->  h [rows x I]           (fp16, in scratch)
//   down:     [128 rows x I] . [I x H]   ->             dm [rows x H]          (fp32, unweighted, row = dispatch slot)
// which is what Basalt's fp4::run_group computes (include/basalt/prefill/moe_fp4.hpp:43-113, src/prefill/moe_fp4.cu:368-518,
// :654-676) - but that kernel is mma.sync kind::mxf4nvf4 for sm_120a, does not assemble for sm_100, and rounds activations
// to FP4.  Here the NVFP4 weights are decoded EXACTLY to fp16 (E2M1 x UE4M3 has at most 5 significant bits) by the producer
// warps straight into 128-byte-swizzled shared memory, activations are fp16 (bf16 inputs convert exactly after a per-row
// power-of-two scale), and tcgen05.mma kind::f16 accumulates in fp32 in tensor memory.  So the result sits ~2e-4 from the
// dequantised fp32 reference instead of the reference kernel's ~1e-2 .. 0.2, at bf16-class tensor throughput.
//
// Persistent CTAs, one per SM, each looping over work items (128-row tile of one expert, 256 weight rows).  Warp roles:
// warp 0 allocates all 512 TMEM columns (two 256-column accumulators) and its lane 0 issues the MMAs (M = 128, N = 256);
// warps 1-2 load the tile's activation rows (cp.async gather through `src`); warps 3-18 decode NVFP4 weight rows to fp16
// straight into 128-byte-swizzled shared memory (two groups of 256 threads, a thread per weight row, the groups taking
// alternate pairs of 64-column k-blocks); warps 19-22 are the epilogue (thread = TMEM lane = output row), which drains one
// accumulator while the tensor core fills the other.  K-blocks move through a ring of four stages (Q6_K three) guarded by mbarriers; every wait
// is bounded and reports through a status word instead of hanging.
//
// Both operands use the SAME permutation of k inside each 16-column group, (0,8,1,9,...,7,15) - the order cvt.e2m1x2 emits
// a sub-block's values in - so no shuffling is needed: the activation image (made by a small kernel here) and the SwiGLU
// output are simply written in that order.
#include <atomic>
#include <type_traits>
#include <cuda_fp16.h>

#include "common.cuh"
#include "experts.cuh"
#include "formats.cuh"
#include "fp16_rows.cuh"
#include "iq1m.cuh"
#include "tc5.cuh"

namespace bsx {
namespace {

constexpr int kTileM = 128;        // rows (tokens) per tile = TMEM lanes
constexpr int kTileN = 256;        // weight rows per tile = TMEM columns of one accumulator
constexpr int kBlockK = 64;        // fp16 per k-block: one 128-byte swizzle row
constexpr int kStagesP = 4;
constexpr int kLoaderWarps = 2, kDecoderWarps = 16, kEpilogueWarps = 4;
constexpr int kGroupThreads = 256; // one group of weight decoders: a thread per weight row of the tile
constexpr int kThreadsP = 32 * (1 + kLoaderWarps + kDecoderWarps + kEpilogueWarps);
constexpr float kHScale = 0.25f;   // the SwiGLU output is stored as fp16(h / 4): fp16 then holds |h| up to 2.6e5

enum { PMODE_GU = 0, PMODE_DOWN = 1 };
enum { WT_NVFP4 = 0, WT_Q6K = 1, WT_IQ1M = 2 };      // how the decoder warps read a weight row
constexpr float kWScaleKQ = 16.f;  // K / I-quant weights are stored as fp16(16 w): typical weights (~1e-2) sit well inside fp16's normal range
enum { kStatusTimeout = 1 };

constexpr uint32_t kInstrDesc = instr_desc_f16(kTileM, kTileN);

__device__ __forceinline__ void cvt_e2m1x8(uint32_t w, uint32_t (&h)[4]) {
    asm("{\n.reg .b8 b0, b1, b2, b3;\nmov.b32 {b0, b1, b2, b3}, %4;\ncvt.rn.f16x2.e2m1x2 %0, b0;\ncvt.rn.f16x2.e2m1x2 %1, b1;\n"
        "cvt.rn.f16x2.e2m1x2 %2, b2;\ncvt.rn.f16x2.e2m1x2 %3, b3;\n}\n"
        : "=r"(h[0]), "=r"(h[1]), "=r"(h[2]), "=r"(h[3])
        : "r"(w));
}
__device__ __forceinline__ uint32_t hmul2_bits(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;\n" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
// UE4M3 byte -> fp16 pair {d, d}, d = scale / 2^8 (see experts_mma.cu: the epilogue multiplies by 2^8); 0x7F -> 0
__device__ __forceinline__ uint32_t scale_pair_bits(uint32_t byte) {
    const uint32_t b = byte & 0x7Fu;
    const uint32_t v = b == 0x7Fu ? 0u : b << 7;
    return v | (v << 16);
}

// IQ1_M weights as fp16(16 w): the exact 8 w / d of iq1m.cuh times 2 d, rounded once, so the stored value is the same fp16 the fp32
// product would round to.  d2: 2 d twice.  out[i] = values i (low half) and i + 8 (high half): the k order both operands are stored in.
__device__ __forceinline__ void iq1m_16(uint32_t q16, uint32_t h8, uint32_t s3, uint32_t d2, const uint16_t* grid, uint32_t (&out)[8]) {
    iq1m_units_16(q16, h8, s3, grid, out);
#pragma unroll
    for (int i = 0; i < 8; ++i) out[i] = hmul2_bits(out[i], d2);
}
// the block's fp16 super-scale times two, in both halves
__device__ __forceinline__ uint32_t iq1m_twice_d(uint2 sc) {
    const uint32_t d = iq1m_d_bits(sc) * 0x10001u;
    return iq1m_add2(d, d);
}

struct PrefillArgs {
    bsx_expert_layout L;
    const unsigned long long* blob_table;   // [E] device addresses
    const int32_t* off;                      // [E + 1] row offsets per expert
    const int32_t* src;                      // [rows] token of each row
    const int32_t* tiles;                    // {expert, first row} per 128-row tile
    const int32_t* n_tiles;
    const __half* xh;                        // [T][H] fp16, permuted, row-scaled
    const float* xinv;                       // [T]
    const uint16_t* grid;                    // the IQ1 codebook on this device
    __half* h;                               // [rows][I] fp16 (permuted, times kHScale)
    float* dm;                               // [rows][H] fp32
    int32_t* status;                         // sticky error word (0 = ok)
};

// Stages: Q6_K gives one up for the raw words of the two decoder groups, half a block of 256 rows each.
template <int WT> constexpr int kStagesOf = WT == WT_Q6K ? kStagesP - 1 : kStagesP;
constexpr int kRawPitch = 31, kRawWords = 256 * kRawPitch;      // 30 words a row; an odd pitch, so that 32 rows' words meet no bank twice
template <int WT>
constexpr size_t kSmemOf = 1024 + kStagesOf<WT> * (kTileM * kBlockK * 2 + kTileN * kBlockK * 2) + 256 + 1024 + 4096 + 64 + (WT == WT_Q6K ? 2 * kRawWords * 4 : 0);
static_assert(kSmemOf<WT_Q6K> <= 227 * 1024 && kSmemOf<WT_NVFP4> <= 227 * 1024, "one CTA per SM");

template <int MODE, bool ALIGNED, int WT>
__global__ void __launch_bounds__(kThreadsP, 1) prefill_gemm_kernel(PrefillArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // 1024-byte aligned operand stages: A then B per stage
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t) 1023);
    constexpr int kABytes = kTileM * kBlockK * 2, kBBytes = kTileN * kBlockK * 2, kStage = kABytes + kBBytes, kStg = kStagesOf<WT>;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kStg * kStage);
    uint64_t* full = bars;                        // [S] loader lanes + one decoder group arrive
    uint64_t* empty = bars + kStg;            // [S] tcgen05.commit arrives
    uint64_t* acc_full = bars + 2 * kStg;     // [2] tcgen05.commit after a tile's last MMA
    uint64_t* acc_empty = acc_full + 2;           // [2] the 128 epilogue threads arrive
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    uint32_t* lut = tmem_slot + 2;                // [256] fp16 scale pairs
    uint16_t* s_grid = reinterpret_cast<uint16_t*>(lut + 256);   // [2048] the IQ1 codebook (IQ1_M rows only)

    // Q6_K: the decoder, which sets the pace there, loses by a warp index from a shuffle (4096 rows of 2048 x 512: 1.919 ms against 1.903)
    const int warp = WT == WT_Q6K ? (int) (threadIdx.x >> 5) : warp_index(), lane = threadIdx.x & 31;
    const int64_t K = MODE == PMODE_GU ? a.L.n_embd : a.L.n_ff;
    const int nkb = (int) (K / kBlockK);
    const int n_out = MODE == PMODE_GU ? (int) a.L.n_ff : (int) a.L.n_embd;      // neurons, or down rows
    constexpr int kOutPerTile = MODE == PMODE_GU ? kTileN / 2 : kTileN;
    const int n_n = (n_out + kOutPerTile - 1) / kOutPerTile;
    const int n_items = *a.n_tiles * n_n;

    for (int i = threadIdx.x; i < 256; i += kThreadsP) lut[i] = scale_pair_bits(i);
    if (WT == WT_IQ1M)
        for (int i = threadIdx.x; i < 2048; i += kThreadsP) s_grid[i] = a.grid[i];
    if (threadIdx.x == 0) {
        for (int s = 0; s < kStg; ++s) {
            mbar_init(&full[s], kGroupThreads + 32 * kLoaderWarps);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], 32 * kEpilogueWarps);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();   // lane 0 initialised the barriers above: reconverge before the warp-wide allocation
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    bool ok = true;

    // A work item: tile = item / n_n (expert, first row), weight rows n0 = (item % n_n) * kOutPerTile ...; every role walks the
    // same item sequence and skips the same items (experts another device holds), so their k-block counters stay in step.
    struct Item { const uint8_t* blob; int row0, rows, n0; };
    auto get_item = [&](int item, Item& it) -> bool {
        const int tile = item / n_n;
        const int expert = a.tiles[2 * tile];
        const unsigned long long bp = a.blob_table[expert];
        if (bp == 0ull) return false;
        it.blob = reinterpret_cast<const uint8_t*>(bp);
        it.row0 = a.tiles[2 * tile + 1];
        it.rows = min(kTileM, a.off[expert + 1] - it.row0);
        it.n0 = (item - tile * n_n) * kOutPerTile;
        return true;
    };

    if (warp == 0) {
        // ---- MMA issuer: one lane feeds the tensor core, four k = 16 instructions per 64-column k-block
        if (elect_one()) {
            uint32_t kc = 0, ti = 0;
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                Item it;
                if (!get_item(item, it)) continue;
                const uint32_t acc = ti & 1u;
                ok = mbar_wait(&acc_empty[acc], ((ti >> 1) & 1u) ^ 1u);     // the epilogue has drained this accumulator
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                for (int kb = 0; kb < nkb; ++kb, ++kc) {
                    const uint32_t s = kc % kStg;
                    ok = mbar_wait(&full[s], (kc / kStg) & 1u);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t sa = smem_u32(smem + s * kStage), sb = sa + kABytes;
                    const uint64_t ad = smem_desc_sw128(sa), bd = smem_desc_sw128(sb);      // addresses in 16 bytes: 2 a step
#pragma unroll
                    for (int k = 0; k < kBlockK / 16; ++k) umma_f16(tmem + acc * kTileN, ad + 2 * k, bd + 2 * k, kInstrDesc, (kb | k) ? 1u : 0u);
                    umma_commit(&empty[s]);      // the stage may be refilled once these MMAs have read it
                }
                if (!ok) break;
                umma_commit(&acc_full[acc]);     // fires when every MMA of the tile has finished
                ++ti;
            }
            if (!ok) atomicOr(a.status, kStatusTimeout);
        }
    } else if (warp <= kLoaderWarps) {
        // ---- activation loaders.  Lane l of loader warp w copies 16-byte chunk l % 8 of rows 64 w + l / 8 + 4 i: eight lanes
        // cover one row's 128 bytes.  Rows past the expert's last row read some valid row instead (never stored).  A lane
        // runs up to two k-blocks ahead of its own completed copies and arrives on a stage once its copies there landed.
        const int lw = warp - 1, c = lane & 7, r4 = lane >> 3;
        const uint8_t* abase = reinterpret_cast<const uint8_t*>(MODE == PMODE_GU ? a.xh : a.h);
        uint32_t dsto[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r7 = 4 * h + r4;
            dsto[h] = (uint32_t) (lw * 8 * 1024 + r7 * 128 + ((c ^ r7) << 4));
        }
        uint32_t issued = 0, arrived = 0;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
            Item it;
            if (!get_item(item, it)) continue;
            uint32_t aoff[16];   // row starts in 16-byte units
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int r = lw * 64 + 4 * i + r4;
                const uint32_t grow = MODE == PMODE_GU ? (uint32_t) a.src[it.row0 + (r < it.rows ? r : 0)] : (uint32_t) (it.row0 + r);
                aoff[i] = grow * (uint32_t) (K >> 3) + (uint32_t) c;
            }
            for (int kb = 0; kb < nkb; ++kb) {
                const uint32_t s = issued % kStg;
                ok = mbar_wait(&empty[s], ((issued / kStg) & 1u) ^ 1u);
                if (!ok) break;
                const uint32_t dst = smem_u32(smem + s * kStage);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const uint8_t* g = abase + ((size_t) aoff[i] + (size_t) kb * 8) * 16;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + (uint32_t) ((i >> 1) * 1024) + dsto[i & 1]), "l"(g) : "memory");
                }
                asm volatile("cp.async.commit_group;\n" ::: "memory");
                ++issued;
                if (issued - arrived > kStg - 2) {      // one less than could be requested, or the tensor core would wait for its own last stage
                    asm volatile("cp.async.wait_group %0;\n" ::"n"(kStg - 2) : "memory");
                    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                    mbar_arrive(&full[arrived % kStg]);
                    ++arrived;
                }
            }
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        for (; arrived < issued; ++arrived) mbar_arrive(&full[arrived % kStg]);
        if (!ok) atomicOr(a.status, kStatusTimeout);
    } else if (warp <= kLoaderWarps + kDecoderWarps) {
        // ---- weight decoders: thread (group, row r) turns the NVFP4 blocks of weight row r of the tile into fp16 B-tile rows
        const int td = threadIdx.x - 32 * (1 + kLoaderWarps);
        const int grp = td >> 8, r = td & 255;
        const uint32_t swz = (uint32_t) (r & 7);
        const uint32_t row_off = (uint32_t) (kABytes + (r >> 3) * 1024 + (r & 7) * 128);
        auto weight_row = [&](const Item& it) -> const uint8_t* {
            if (MODE == PMODE_GU) {     // B rows 0..127 = gate rows, 128..255 = the matching up rows
                const int n = min(it.n0 + (r & 127), n_out - 1);
                return r < 128 ? it.blob + (size_t) n * a.L.gu_row : it.blob + a.L.up_off + (size_t) n * a.L.up_row;
            }
            return it.blob + a.L.down_off + (size_t) min(it.n0 + r, n_out - 1) * a.L.d_row;
        };
        // one NVFP4 block (9 words: 4 scale bytes, 32 code bytes) -> 64 fp16 of the B tile, already in the permuted k order
        auto store_b = [&](uint32_t s, const uint32_t* cur) {
            uint4* brow = reinterpret_cast<uint4*>(smem + s * kStage + row_off);
#pragma unroll
            for (int sub = 0; sub < 4; ++sub) {
                const uint32_t sc = lut[(cur[0] >> (8 * sub)) & 0xFFu];
                uint32_t q0[4], q1[4];
                cvt_e2m1x8(cur[1 + 2 * sub], q0);
                cvt_e2m1x8(cur[2 + 2 * sub], q1);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    q0[i] = hmul2_bits(q0[i], sc);
                    q1[i] = hmul2_bits(q1[i], sc);
                }
                brow[(2 * sub) ^ swz] = make_uint4(q0[0], q0[1], q0[2], q0[3]);
                brow[(2 * sub + 1) ^ swz] = make_uint4(q1[0], q1[1], q1[2], q1[3]);
            }
        };
        // the pair of blocks q (k-blocks 2q, 2q + 1): 72 bytes at offset 72 q of the row; 16-byte loads when rows are whole
        // 144-byte chunks (then 72 q is a multiple of 16 for even q and of 8 for odd q)
        const int npair = (nkb + 1) >> 1;
        auto load_pair = [&](const uint8_t* wrow, int q, uint32_t (&w)[18]) {
            const uint8_t* src = wrow + (size_t) q * 72;
            if (ALIGNED) {
                if ((q & 1) == 0) {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint4 v = reinterpret_cast<const uint4*>(src)[i];
                        w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
                    }
                    const uint2 t = reinterpret_cast<const uint2*>(src)[8];
                    w[16] = t.x; w[17] = t.y;
                } else {
                    const uint2 t = reinterpret_cast<const uint2*>(src)[0];
                    w[0] = t.x; w[1] = t.y;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint4 v = reinterpret_cast<const uint4*>(src + 8)[i];
                        w[2 + 4 * i] = v.x; w[3 + 4 * i] = v.y; w[4 + 4 * i] = v.z; w[5 + 4 * i] = v.w;
                    }
                }
            } else {
                const int nw = 2 * q + 1 < nkb ? 18 : 9;
#pragma unroll
                for (int i = 0; i < 18; ++i) w[i] = i < nw ? reinterpret_cast<const uint32_t*>(src)[i] : 0u;
            }
        };
        if constexpr (WT == WT_NVFP4) {
            // the stream of own pairs runs across items: the first pair of the next item is requested while the last pair of this
            // one is decoded, so a tile switch does not expose a load
            uint32_t wc[18], wn[18];
            // The groups take turns across items too (an item may have an odd number of pairs): a group that left out more k-blocks than there
            // are stages could take an earlier phase of a stage's barrier for the one it waits for.
            uint32_t kc = 0;
            int first = grp;
            int item = blockIdx.x;
            Item it;
            while (item < n_items && !get_item(item, it)) item += gridDim.x;
            if (item < n_items && first < npair) load_pair(weight_row(it), first, wn);
            while (item < n_items && ok) {
                const uint8_t* wrow = weight_row(it);
                int nxt = item + gridDim.x;
                Item itn;
                while (nxt < n_items && !get_item(nxt, itn)) nxt += gridDim.x;
                const int first_next = first ^ (npair & 1);
                for (int q = first; q < npair && ok; q += 2) {
#pragma unroll
                    for (int i = 0; i < 18; ++i) wc[i] = wn[i];
                    if (q + 2 < npair) load_pair(wrow, q + 2, wn);
                    else if (nxt < n_items && first_next < npair) load_pair(weight_row(itn), first_next, wn);
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int kb = 2 * q + j;
                        if (kb < nkb && ok) {
                            const uint32_t kk = kc + (uint32_t) kb, s = kk % kStg;
                            ok = mbar_wait(&empty[s], ((kk / kStg) & 1u) ^ 1u);
                            if (ok) {
                                store_b(s, &wc[9 * j]);
                                asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");   // generic-proxy writes -> visible to the tensor core
                                mbar_arrive(&full[s]);
                            }
                        }
                    }
                }
                if (first >= npair && nxt < n_items && first_next < npair) load_pair(weight_row(itn), first_next, wn);      // this item had no pair for the group
                first = first_next;
                kc += (uint32_t) nkb;
                item = nxt;
                it = itn;
            }
        } else if constexpr (WT == WT_IQ1M) {
            // IQ1_M rows: half a block (128 values: 16 index bytes, 8 bytes of high bits, the 8 scale bytes) is one pair of k-blocks.
            // The next half is requested before this one is decoded, across items too; the decode runs ahead of the wait for the
            // stage, so it overlaps the tensor core.
            uint2 nx[4];
            auto load_half = [&](const uint8_t* wrow, int q) {
                const uint8_t* blk = wrow + (size_t) (q >> 1) * 56;
                const int hb = q & 1;
                nx[0] = *reinterpret_cast<const uint2*>(blk + 16 * hb);
                nx[1] = *reinterpret_cast<const uint2*>(blk + 16 * hb + 8);
                nx[2] = *reinterpret_cast<const uint2*>(blk + 32 + 8 * hb);
                nx[3] = *reinterpret_cast<const uint2*>(blk + 48);
            };
            uint32_t kc = 0;
            int item = blockIdx.x;
            Item it;
            while (item < n_items && !get_item(item, it)) item += gridDim.x;
            if (item < n_items && grp < npair) load_half(weight_row(it), grp);
            while (item < n_items && ok) {
                const uint8_t* wrow = weight_row(it);
                int nxt = item + gridDim.x;
                Item itn;
                while (nxt < n_items && !get_item(nxt, itn)) nxt += gridDim.x;
                for (int q = grp; q < npair && ok; q += 2) {
                    const uint32_t qs[4] = {nx[0].x, nx[0].y, nx[1].x, nx[1].y}, qh[2] = {nx[2].x, nx[2].y};
                    const uint2 sc = nx[3];
                    if (q + 2 < npair) load_half(wrow, q + 2);
                    else if (nxt < n_items) load_half(weight_row(itn), grp);
                    const uint32_t d2 = iq1m_twice_d(sc);
                    const uint32_t scw = (q & 1) ? sc.y : sc.x;
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const int kb = 2 * q + j;
                        uint32_t p[4][8];
#pragma unroll
                        for (int sub = 0; sub < 4; ++sub)
                            iq1m_16((qs[2 * j + (sub >> 1)] >> (16 * (sub & 1))) & 0xFFFFu, (qh[j] >> (8 * sub)) & 0xFFu, (scw >> (16 * j + 3 * sub)) & 7u, d2, s_grid, p[sub]);
                        const uint32_t kk = kc + (uint32_t) kb, s = kk % kStg;
                        ok = mbar_wait(&empty[s], ((kk / kStg) & 1u) ^ 1u);
                        if (!ok) break;
                        uint4* brow = reinterpret_cast<uint4*>(smem + s * kStage + row_off);
#pragma unroll
                        for (int sub = 0; sub < 4; ++sub) {
                            brow[(2 * sub) ^ swz] = make_uint4(p[sub][0], p[sub][1], p[sub][2], p[sub][3]);
                            brow[(2 * sub + 1) ^ swz] = make_uint4(p[sub][4], p[sub][5], p[sub][6], p[sub][7]);
                        }
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                        mbar_arrive(&full[s]);
                    }
                }
                kc += (uint32_t) nkb;
                item = nxt;
                it = itn;
            }
        } else {
            // Q6_K rows (210 bytes per 256 values, on 2 bytes): a pair of k-blocks is half a block - 64 bytes of low bits, 32 of high bits, 8
            // scales, d - as the 30 words that cover it, which the group's warps fetch row by row (a row's words side by side, where a
            // thread reading its own row touches 32 lines a load) into shared memory.  A thread then decodes its row: codes four at a
            // time, each to fp32 by its byte under the exponent of 2^23, times 16 d sc, pairs rounded to fp16 - the only rounding, 2^-11
            // relative.  4096 rows of 2048 x 512, 512 experts, whole layer: byte by byte from global memory 28.4 ms, so 1.94.
            // A wait that gave up does not end the loop: the other threads of the group wait for this one at its barriers.
            uint32_t* raw = reinterpret_cast<uint32_t*>(s_grid + 2048) + grp * kRawWords;
            const uint32_t* mine = raw + r * kRawPitch;
            const int warp_g = td >> 5 & 7;
            const int seg = lane < 17 ? 0 : lane < 26 ? 1 : lane < 29 ? 2 : 3, seg_word = lane - (seg == 0 ? 0 : seg == 1 ? 17 : seg == 2 ? 26 : 29);
            uint32_t kc = 0;
            for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
                Item it;
                if (!get_item(item, it)) continue;
                auto row_at = [&](int row) -> const uint8_t* {
                    if (MODE == PMODE_GU) {
                        const int n = min(it.n0 + (row & 127), n_out - 1);
                        return row < 128 ? it.blob + (size_t) n * a.L.gu_row : it.blob + a.L.up_off + (size_t) n * a.L.up_row;
                    }
                    return it.blob + a.L.down_off + (size_t) min(it.n0 + row, n_out - 1) * a.L.d_row;
                };
                const bool own_odd = (reinterpret_cast<uintptr_t>(row_at(r)) & 2) != 0;
                for (int q = grp; q < npair; q += 2) {
                    const size_t blk = (size_t) (q >> 1) * 210;
                    const int hb = q & 1;
                    const size_t off = blk + (seg == 0 ? 64 * hb : seg == 1 ? 128 + 32 * hb : seg == 2 ? 192 + 8 * hb : 208);
                    asm volatile("bar.sync %0, 256;\n" ::"r"(1 + grp) : "memory");            // everyone is done with the words of the pair before
#pragma unroll 4
                    for (int i = 0; i < 32; ++i) {
                        const int row = 32 * warp_g + i;
                        const uintptr_t src = (reinterpret_cast<uintptr_t>(row_at(row) + off) & ~(uintptr_t) 3) + 4 * seg_word;
                        if (lane < 30)
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(smem_u32(raw + row * kRawPitch + lane)), "l"(src) : "memory");
                    }
                    asm volatile("cp.async.wait_all;\n" ::: "memory");
                    asm volatile("bar.sync %0, 256;\n" ::"r"(1 + grp) : "memory");
                    const bool odd = own_odd != ((q >> 1) & 1);
                    auto word = [&](int first, int k) { return odd ? __funnelshift_r(mine[first + k], mine[first + k + 1], 16) : mine[first + k]; };
                    const uint32_t dw = mine[29];
                    const float d16 = __half2float(__ushort_as_half((unsigned short) (odd ? dw >> 16 : dw & 0xFFFFu))) * kWScaleKQ;
                    const uint32_t sc[2] = {word(26, 0), word(26, 1)};
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint32_t kk = kc + (uint32_t) (2 * q + j), s = kk % kStg;
                        if (ok) ok = mbar_wait(&empty[s], ((kk / kStg) & 1u) ^ 1u);
                        uint4* brow = reinterpret_cast<uint4*>(smem + s * kStage + row_off);
#pragma unroll
                        for (int sub = 0; sub < 4; ++sub) {
                            const int g4 = 4 * j + sub, from = g4 >> 1, l16 = g4 & 1;             // 32 values `from` of the half, 16 of them
                            const float scale = d16 * (float) (int8_t) (sc[g4 >> 2] >> (8 * (g4 & 3)));
                            uint32_t c[4];
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const uint32_t lo = word(0, (from & 1) * 8 + 4 * l16 + i), hi = word(17, 4 * l16 + i);
                                c[i] = ((from >= 2 ? lo >> 4 : lo) & 0x0F0F0F0Fu) | (((hi >> (2 * from)) & 0x03030303u) << 4);
                            }
                            uint32_t p[8];
#pragma unroll
                            for (int i = 0; i < 8; ++i) {       // values i and i + 8: the k order both operands are stored in
                                const float u = __uint_as_float(__byte_perm(c[i >> 2], 0x4B000000u, 0x7440 + (i & 3))) - 8388640.f;
                                const float v = __uint_as_float(__byte_perm(c[2 + (i >> 2)], 0x4B000000u, 0x7440 + (i & 3))) - 8388640.f;
                                const __half2 h2 = __floats2half2_rn(u * scale, v * scale);
                                p[i] = *reinterpret_cast<const uint32_t*>(&h2);
                            }
                            if (ok) {
                                brow[(2 * sub) ^ swz] = make_uint4(p[0], p[1], p[2], p[3]);
                                brow[(2 * sub + 1) ^ swz] = make_uint4(p[4], p[5], p[6], p[7]);
                            }
                        }
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                        if (ok) mbar_arrive(&full[s]);
                    }
                }
                kc += (uint32_t) nkb;
            }
        }
        if (!ok) atomicOr(a.status, kStatusTimeout);
    } else {
        // ---- epilogue: thread p reads TMEM lane p (= output row p) of the finished accumulator.  A warp may only read the 32
        // TMEM lanes 32 (warp % 4) .. + 31.  tcgen05.ld is warp-wide: every lane runs the loads; only the stores are predicated.
        const int p = (warp & 3) * 32 + lane;
        const uint32_t lane_base = (uint32_t) ((warp & 3) * 32) << 16;
        const int form = swiglu_form(a.L);
        uint32_t ti = 0;
        for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
            Item it;
            if (!get_item(item, it)) continue;
            const uint32_t acc = ti & 1u;
            ok = __all_sync(kFull, mbar_wait(&acc_full[acc], (ti >> 1) & 1u));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const bool row_live = p < it.rows;
            // NVFP4 blobs end in {s_gate, s_up, s_down, 0}; the block scales were used as scale / 2^8.  K / I-quant rows have no
            // tail and were stored as 16 w.
            const bool nv_tail = a.L.gu_type == kTypeNVFP4;
            const float* tail = reinterpret_cast<const float*>(it.blob + a.L.bytes - 16);
            constexpr float kUnscale = WT == WT_NVFP4 ? 256.f : 1.f / kWScaleKQ;
            const uint32_t tbase = tmem + lane_base + acc * kTileN;
            if (MODE == PMODE_GU) {
                const float f = row_live ? a.xinv[a.src[it.row0 + p]] * kUnscale : 0.f;
                const float sg = (nv_tail ? tail[0] : 1.f) * f, su = (nv_tail ? tail[1] : 1.f) * f;
                __half* hrow = a.h + (size_t) (it.row0 + p) * a.L.n_ff + it.n0;
#pragma unroll 1
                for (int c0 = 0; c0 < kTileN / 2; c0 += 16) {
                    uint32_t g[16], u[16];
                    tmem_ld16(tbase + (uint32_t) c0, g);
                    tmem_ld16(tbase + (uint32_t) (kTileN / 2 + c0), u);
                    __half out[16];
                    auto work = [&](auto act) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const float hv = swiglu_as<decltype(act)::value>(__uint_as_float(g[j]) * sg, __uint_as_float(u[j]) * su, a.L) * kHScale;
                            out[perm16(j)] = __float2half_rn(fminf(fmaxf(hv, -65504.f), 65504.f));
                        }
                    };
                    if (form == SWIGLU_PLAIN) work(std::integral_constant<int, SWIGLU_PLAIN>{});
                    else if (form == SWIGLU_LIMIT) work(std::integral_constant<int, SWIGLU_LIMIT>{});
                    else work(std::integral_constant<int, SWIGLU_CAP>{});
                    if (row_live && it.n0 + c0 < n_out) {
                        reinterpret_cast<uint4*>(hrow + c0)[0] = reinterpret_cast<const uint4*>(out)[0];
                        reinterpret_cast<uint4*>(hrow + c0)[1] = reinterpret_cast<const uint4*>(out)[1];
                    }
                }
            } else {
                const float f = (nv_tail ? tail[2] : 1.f) * (kUnscale / kHScale);
                float* orow = a.dm + (size_t) (it.row0 + p) * a.L.n_embd + it.n0;
#pragma unroll 1
                for (int c0 = 0; c0 < kTileN; c0 += 32) {
                    uint32_t d[32];
                    tmem_ld32(tbase + (uint32_t) c0, d);
                    if (row_live && it.n0 + c0 < n_out) {
#pragma unroll
                        for (int v = 0; v < 8; ++v)
                            reinterpret_cast<float4*>(orow + c0)[v] = make_float4(__uint_as_float(d[4 * v]) * f, __uint_as_float(d[4 * v + 1]) * f,
                                                                                 __uint_as_float(d[4 * v + 2]) * f, __uint_as_float(d[4 * v + 3]) * f);
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            mbar_arrive(&acc_empty[acc]);
            ++ti;
        }
        if (!ok && lane == 0) atomicOr(a.status, kStatusTimeout);
    }
    // everyone is done with tensor memory before warp 0 gives it back
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
    }
}

size_t align256p(size_t v) { return (v + 255) & ~(size_t) 255; }

int wt_of(int type) { return type == kTypeNVFP4 ? WT_NVFP4 : type == kTypeQ6K ? WT_Q6K : type == kTypeIQ1M ? WT_IQ1M : -1; }

template <int MODE, bool ALIGNED, int WT>
cudaError_t configure_one() { return cudaFuncSetAttribute(prefill_gemm_kernel<MODE, ALIGNED, WT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) kSmemOf<WT>); }

template <int MODE>
void launch_mode(int wt, bool aligned16, unsigned grid, const PrefillArgs& a, cudaStream_t st) {
    if (wt == WT_NVFP4) {
        if (aligned16) prefill_gemm_kernel<MODE, true, WT_NVFP4><<<grid, kThreadsP, kSmemOf<WT_NVFP4>, st>>>(a);
        else prefill_gemm_kernel<MODE, false, WT_NVFP4><<<grid, kThreadsP, kSmemOf<WT_NVFP4>, st>>>(a);
    } else if (wt == WT_Q6K) {
        prefill_gemm_kernel<MODE, false, WT_Q6K><<<grid, kThreadsP, kSmemOf<WT_Q6K>, st>>>(a);
    } else {
        prefill_gemm_kernel<MODE, false, WT_IQ1M><<<grid, kThreadsP, kSmemOf<WT_IQ1M>, st>>>(a);
    }
}

}  // namespace
}  // namespace bsx

using namespace bsx;

extern "C" size_t bsx_experts_prefill_scratch_bytes(const bsx_expert_layout* L, int64_t n_tokens, int64_t cap_rows) {
    if (!L || n_tokens < 0 || cap_rows < 0) return 0;
    return align256p((size_t) n_tokens * L->n_embd * 2) + align256p((size_t) n_tokens * 4) + align256p((size_t) (cap_rows + kTileM) * L->n_ff * 2) + 256;
}

extern "C" int32_t bsx_experts_prefill(const bsx_expert_layout* layout, const unsigned long long* blob_table, const int32_t* off,
                                       const int32_t* src, const int32_t* tiles, const int32_t* n_tiles, int64_t cap_tiles, int64_t cap_rows,
                                       const void* x, int32_t x_kind, int64_t n_tokens, void* scratch, float* dm, int32_t* status, void* stream) {
    if (!stream) return BSX_E_STREAM;
    if (!layout || !blob_table || !off || !src || !tiles || !n_tiles || !aligned(x, 16) || !aligned(scratch, 256) || !aligned(dm, 16) || !status)
        return BSX_E_POINTER;
    const bsx_expert_layout& L = *layout;
    const int wt_gu = wt_of(L.gu_type), wt_d = wt_of(L.d_type);
    if (wt_gu < 0 || wt_d < 0 || L.up_type != L.gu_type) return BSX_E_TYPE;       // NVFP4, Q6_K or IQ1_M; gate and up of one format
    if ((L.gu_type == kTypeNVFP4) != (L.d_type == kTypeNVFP4) && L.gu_type == kTypeNVFP4) return BSX_E_TYPE;   // an NVFP4 tail needs NVFP4 gate / up
    if (L.n_embd % 64 || L.n_ff % 64 || (x_kind != BSX_X_F32 && x_kind != BSX_X_BF16)) return BSX_E_GEOMETRY;
    if ((wt_gu != WT_NVFP4 && L.n_embd % 256) || (wt_d != WT_NVFP4 && L.n_ff % 256)) return BSX_E_GEOMETRY;   // whole 256-value blocks
    if (cap_tiles < 0 || cap_tiles > 65535 || cap_rows < 0 || n_tokens < 0) return BSX_E_GEOMETRY;
    if (cap_tiles == 0 || n_tokens == 0) return BSX_OK;
    const cudaStream_t st = (cudaStream_t) stream;
    uint8_t* p = static_cast<uint8_t*>(scratch);
    PrefillArgs a;
    a.L = L;
    a.blob_table = blob_table;
    a.off = off;
    a.src = src;
    a.tiles = tiles;
    a.n_tiles = n_tiles;
    __half* xh = reinterpret_cast<__half*>(p);
    p += align256p((size_t) n_tokens * L.n_embd * 2);
    float* xinv = reinterpret_cast<float*>(p);
    p += align256p((size_t) n_tokens * 4);
    a.xh = xh;
    a.xinv = xinv;
    a.grid = iq1_device_grid();
    if (!a.grid) return (int32_t) cudaErrorInvalidSymbol;
    a.h = reinterpret_cast<__half*>(p);
    a.dm = dm;
    a.status = status;
    static std::atomic<bool> configured[64];   // per device; threads of different devices call concurrently
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return (int32_t) cudaErrorInvalidDevice;
    if (!configured[dev].load(std::memory_order_acquire)) {
        cudaError_t e = configure_one<PMODE_GU, true, WT_NVFP4>();
        if (e == cudaSuccess) e = configure_one<PMODE_GU, false, WT_NVFP4>();
        if (e == cudaSuccess) e = configure_one<PMODE_DOWN, true, WT_NVFP4>();
        if (e == cudaSuccess) e = configure_one<PMODE_DOWN, false, WT_NVFP4>();
        if (e == cudaSuccess) e = configure_one<PMODE_GU, false, WT_Q6K>();
        if (e == cudaSuccess) e = configure_one<PMODE_DOWN, false, WT_Q6K>();
        if (e == cudaSuccess) e = configure_one<PMODE_GU, false, WT_IQ1M>();
        if (e == cudaSuccess) e = configure_one<PMODE_DOWN, false, WT_IQ1M>();
        if (e != cudaSuccess) return (int32_t) e;
        configured[dev].store(true, std::memory_order_release);
    }
    const PlaneRows xr{x, x_kind, 1, n_tokens, xh, xinv}, none{x, x_kind, 1, 0, xh, xinv};
    if (L.n_embd <= 4096) rows_to_fp16_planes_kernel<128><<<(unsigned) ((n_tokens + 1) / 2), 256, 0, st>>>(xr, none, L.n_embd);
    else rows_to_fp16_planes_kernel<256><<<(unsigned) n_tokens, 256, 0, st>>>(xr, none, L.n_embd);
    // persistent CTAs, one per SM; rows that are whole 144-byte chunks (K % 256 == 0) take the variant with 16-byte weight loads
    const unsigned grid = (unsigned) sm_count();
    launch_mode<PMODE_GU>(wt_gu, L.n_embd % 256 == 0, grid, a, st);
    launch_mode<PMODE_DOWN>(wt_d, L.n_ff % 256 == 0, grid, a, st);
    return launch_status();
}
