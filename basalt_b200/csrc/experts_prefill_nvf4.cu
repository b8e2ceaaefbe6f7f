// experts_prefill_nvf4.cu - prompt-sized grouped experts on the block-scaled FP4 tensor cores (tcgen05 kind::mxf4nvf4), over
// blobs packed by bsx_expert_pack.
//
// The same ragged grouped GEMM as experts_prefill.cu (Basalt's fp4::run_group, include/basalt/prefill/moe_fp4.hpp:43-113):
//   gate/up:  [128 rows x H] . [H x 2I]  -> SwiGLU ->  h [rows x I]       (fp32, in scratch)
//   down:     [128 rows x I] . [I x H]   ->             dm [rows x H]      (fp32, unweighted, row = dispatch slot)
// but nothing is decoded: a packed block (128 weight rows x 256 columns: 16 KB of codes in the swizzled order of a stage,
// 2 KB of UE4M3 scale words) is one bulk copy into shared memory and the tensor core reads it as it is.  Activations enter
// as four FP4 terms per row (nvf4.cuh; relative error ~1e-4), i.e. four MMAs per 64-column K-step into one accumulator.
// That is what Basalt's sm_120 kernel does with ONE term (and an optional second) at ~1e-1 .. 1e-2; four terms cost the
// tensor time of an fp16 product and meet the 2e-3 bar.
//
// The products run on pairs of SMs (prefill_pair_kernel).  What was found on the way, gate/up product of the 7168 x 2048 layer at 8192 tokens
// (256 experts + the shared one): one SM a tile, rows gathered, MMAs issued under `lane == 0` 4.88 ms, under elect.sync (tc5.cuh) 3.52;
// pairs 3.14, at 1.36 GHz: the tensor pipe is busy 85 % of the time and the power limit sets the clock.  2048 x 512 at 16,384 tokens, whole
// layer: 2.03 -> 1.67 ms; 4000 rows of 5120 x 2304: 3.7 -> 2.7, for a tile costs what its rows do.
#include <algorithm>
#include <atomic>
#include <type_traits>
#include <cuda_fp16.h>

#include "common.cuh"
#include "experts.cuh"
#include "nvf4.cuh"
#include "pdl.cuh"
#include "plan.cuh"
#include "tc5.cuh"

namespace bsx {

void packed_x_images(const void* x, int kind, int64_t rows, int64_t K, uint8_t* codes, uint8_t* sfs, float* inv, cudaStream_t st);
void packed_listed_images(const float* h, const PassRec* items, const int* n_items, int pass_entries, const TileRec* recs, const int32_t* n_recs, int64_t K, uint8_t* codes,
                          uint8_t* sfs, float* inv, cudaStream_t st);
int32_t packed_pass_product(bool down, const ExpertArgs& a, const PassRec* items, const int* n_items, int pass_entries, const uint8_t* codes, const uint8_t* sfs,
                            const float* inv, int32_t* status, cudaStream_t st);

namespace {

constexpr int kATileQ = 128 * 128;                 // code tile of 128 rows x 256 columns
enum { QMODE_GU = 0, QMODE_DOWN = 1 };

// Tile images, of the SwiGLU rows of long calls.  The rows a tile multiplies lie as a stage has them in shared memory: for each
// (chunk of 256 columns, FP4 term) one run of [2 KB scale words, as tensor memory has them for 128 rows | 1 KB per eight rows of
// codes, 128-byte swizzled], so that a slot is one or two bulk copies.  A tile takes `units` = ceil(rows / 8) + 2 KB per (chunk, term); rows and
// scale words past its last row are never written (each only reaches its own accumulator column, which is not stored).
constexpr int kSFQ = 4 * 512;                      // the scale words: four K-steps of 32 lanes x 4 words
__host__ __device__ __forceinline__ int tile_units(int rows) { return (rows + 7) / 8 + 2; }
__device__ __forceinline__ size_t image_block(const TileRec& r, int n_chunk, int c, int t) {
    return ((size_t) r.base * n_chunk * kTermsF + (size_t) (c * kTermsF + t) * tile_units(r.rows)) * 1024;
}
// units that cap_rows rows in cap_tiles tiles can take
__host__ __device__ inline int64_t image_units(int64_t cap_rows, int64_t cap_tiles) { return cap_rows / 8 + 3 * cap_tiles; }

// The tile list without the tiles of experts held elsewhere.  One block; a scan carries units (or passes) and places together.  Tiles that
// overlap (no dispatch makes them) and exceed the room are left out and set the status word.
// items (optional, a short call): the rows become passes of up to pass_entries rows for the decode stream instead.  But a call that is
// short by its average may still send most rows to a few experts, and the stream reads an expert's weights once a pass: tiles of more
// than kCrowdedRows rows then stay tiles, provided the passes they save outweigh what the tile kernels take in the whole.  A tile costs
// the chip three to four passes (5120 x 2304: 5.5 us of 64 rows, 7.5 of 128, a pass of 16 rows 2.0), and the tile kernels come in rounds of
// items, one a pair of SMs, of which a call pays one more than it fills (launches, the last item's latency).  A third of the rows on a few
// of 385 experts, 16 rows an expert on average, all passes against this rule: on 64 experts 1440 : 1409 us, on 16 1425 : 1357, but on 4
// 1434 : 1503 and on one 1408 : 1556, where it is too willing.
constexpr int kCrowdedRows = 64;
struct RecordArgs {
    const int32_t *tiles, *n_tiles, *off;
    const unsigned long long* blob_table;
    int64_t cap_tiles;
    TileRec* recs;
    int64_t cap_recs;
    int32_t* n_recs;                             // [3]: tiles listed; two counters of the products, zeroed here
    int64_t cap_units;                           // of the tile images
    PassRec* items;
    int* n_items;
    int64_t cap_items;
    int pass_entries, tile_items, sm_count;      // tile_items: SMs that a tile's gate/up product keeps for an item's time (two an item of 256 neurons)
    int32_t* status;
};
__global__ void __launch_bounds__(1024) tile_records_kernel(RecordArgs a) {
    __shared__ unsigned long long sh[32];
    __shared__ unsigned s_end;                                           // tiles from here on have no room
    constexpr unsigned long long kLow = (1ull << 36) - 1;               // units or passes | tiles << 36
    if (threadIdx.x == 0) s_end = (unsigned) a.cap_recs;
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();
    const int64_t n = min(a.cap_tiles, (int64_t) *a.n_tiles);
    auto record = [&](int64_t t) {
        TileRec r = {0ull, 0, 0, 0, 0};
        if (t < n) {
            const int expert = a.tiles[2 * t], row0 = a.tiles[2 * t + 1];
            r.blob = a.blob_table[expert];
            r.row0 = row0;
            r.rows = r.blob != 0ull ? max(0, min(128, a.off[expert + 1] - row0)) : 0;
        }
        return r;
    };
    int tile_rows = 1;                                                   // from this many rows on a tile stays one
    if (a.items) {
        unsigned long long v = 0, total = 0;
        for (int64_t t = threadIdx.x; t < n; t += 1024) {
            const int rows = record(t).rows;
            if (rows > kCrowdedRows) v += (unsigned long long) ((rows + 15) / 16) | (1ull << 36);
        }
        block_excl_sum<unsigned long long>(v, &total, sh);
        const int64_t saved = (int64_t) (total & kLow) * a.tile_items, rounds = ((int64_t) (total >> 36) * a.tile_items + a.sm_count - 1) / a.sm_count;
        tile_rows = saved > 3 * (int64_t) a.sm_count * (rounds + 1) ? kCrowdedRows + 1 : 129;
    }
    int64_t low = 0, placed = 0;
    for (int64_t t0 = 0; t0 < n; t0 += 1024) {
        TileRec r = record(t0 + threadIdx.x);
        const bool tile = r.rows >= tile_rows;
        const int passes = a.items && !tile ? (r.rows + a.pass_entries - 1) / a.pass_entries : 0, u = tile && !a.items ? tile_units(r.rows) : 0;
        unsigned long long total = 0;
        const unsigned long long before = block_excl_sum<unsigned long long>((unsigned long long) (passes + u) | ((unsigned long long) tile << 36), &total, sh);
        const int64_t at = low + (int64_t) (before & kLow), place = placed + (int64_t) (before >> 36);
        low += (int64_t) (total & kLow);
        placed += (int64_t) (total >> 36);
        for (int p = 0; p < passes; ++p) {
            PassRec q;
            q.blob = r.blob;
            q.eb = r.row0 + p * a.pass_entries;
            q.ntok = min(a.pass_entries, r.rows - p * a.pass_entries);
            if (at + p < a.cap_items) a.items[at + p] = q;
        }
        if (!tile) continue;
        if (!a.items) r.base = at;
        if (place < a.cap_recs) a.recs[place] = r;
        if (!a.items && at + u > a.cap_units && place < a.cap_recs) atomicMin(&s_end, (unsigned) place);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (placed > (int64_t) s_end || (a.items && low > a.cap_items)) atomicOr(a.status, 1);
        if (a.items) *a.n_items = (int) min(low, a.cap_items);
        a.n_recs[0] = (int) min(placed, (int64_t) s_end);
        a.n_recs[1] = a.n_recs[2] = 0;
    }
}

struct PrefillFArgs {
    bsx_expert_layout L;
    const TileRec* recs;
    const int32_t* n_recs;
    const int32_t* src;                      // [rows] token of each row
    const uint8_t *img, *sfs;                // the row images of this product's operand: codes, scales
    const float* inv;
    float* h;                                // [rows + 128][I] fp32 SwiGLU output
    float* dm;                               // [rows][H] fp32
    int32_t* status;
    int32_t* counter;                        // of the items drawn in this launch
};

__device__ __forceinline__ void bulk_copy_q(uint32_t dst, const uint8_t* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void expect_bytes_q(uint32_t bar, uint32_t bytes) {
    asm volatile("{\n.reg .b64 t;\nmbarrier.arrive.expect_tx.shared::cta.b64 t, [%0], %1;\n}\n" ::"r"(bar), "r"(bytes) : "memory");
}
constexpr uint64_t kStepCode = 2;                  // descriptors count addresses in 16 bytes: a K-step further is 32 bytes of codes
// rows of h (fp32, dispatch order) -> tile images of the down product.  Block = eight rows of a tile, a warp a row: a lane makes
// one sub-block of 16 values at a time, and four lanes' scale bytes make a word.  NIT = 1: a lane's one sub-block
// stays in registers between the row's maximum and its codes (n_ff <= 512: 205 -> 174 us for 180,224 rows of 512); 0 reads the row
// twice (four sub-blocks in registers were slower there: 274 -> 340 us for 73,728 rows of 2048).
template <int NIT>
__global__ void __launch_bounds__(256) h_images_kernel(const TileRec* recs, const int32_t* n_recs, const float* h, int64_t K,
                                                       uint8_t* __restrict__ img, float* __restrict__ inv) {
    pdl_wait();
    pdl_launch_dependents();
    const int tile = (int) (blockIdx.x >> 4), row = (blockIdx.x & 15) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (tile >= *n_recs) return;
    const TileRec r = recs[tile];
    if (row >= r.rows) return;
    const int64_t i = r.row0 + row;
    const int n_sb = (int) (K >> 4), n_chunk = (int) (K >> 8);
    float amax = 0.f;
    float keep[NIT > 0 ? NIT : 1][16];
    auto load = [&](int sb, float (&v)[16]) {
        if (sb < n_sb) {
            load16(h, BSX_X_F32, i, K, sb, v);
        } else {
#pragma unroll
            for (int j = 0; j < 16; ++j) v[j] = 0.f;
        }
    };
    if constexpr (NIT > 0) {
#pragma unroll
        for (int q = 0; q < NIT; ++q) load(32 * q + lane, keep[q]);
#pragma unroll
        for (int q = 0; q < NIT; ++q)
#pragma unroll
            for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(keep[q][j]));
    } else {
        for (int sb = lane; sb < n_sb; sb += 32) {
            load(sb, keep[0]);
#pragma unroll
            for (int j = 0; j < 16; ++j) amax = fmaxf(amax, fabsf(keep[0][j]));
        }
    }
    amax = warp_max_xor(amax);
    const Pow2Scale ps = fp4_row_scale(amax);
    if (lane == 0) inv[i] = ps.inv;
    const size_t term_bytes = (size_t) tile_units(r.rows) * 1024;
    auto write = [&](int sb, float (&v)[16]) {           // n_sb is a multiple of 16: whole chunks, four lanes of a word together
        const bool live = sb < n_sb;
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] *= ps.s;
        uint8_t* out = img + image_block(r, n_chunk, sb >> 4, 0);
        const int q = sb & 15;
#pragma unroll
        for (int t = 0; t < kTermsF; ++t) {
            uint32_t w0, w1;
            uint32_t sc = fp4_term(v, w0, w1) << (8 * (lane & 3));
            sc |= __shfl_xor_sync(kFull, sc, 1);
            sc |= __shfl_xor_sync(kFull, sc, 2);
            if (!live) continue;
            uint8_t* o = out + t * term_bytes;
            *reinterpret_cast<uint2*>(o + kSFQ + (row >> 3) * 1024 + (row & 7) * 128 + (((q >> 1) ^ (row & 7)) << 4) + (q & 1) * 8) = make_uint2(w0, w1);
            if ((lane & 3) == 0) *reinterpret_cast<uint32_t*>(o + (q >> 2) * 512 + (row & 31) * 16 + (row >> 5) * 4) = sc;
        }
    };
    if constexpr (NIT > 0) {
#pragma unroll
        for (int q = 0; q < NIT; ++q) write(32 * q + lane, keep[q]);
    } else {
        for (int sb = lane; sb - lane < n_sb; sb += 32) {
            load(sb, keep[0]);
            write(sb, keep[0]);
        }
    }
}

// ---------------------------------------------------------------- the products: pairs of SMs
// A pair of CTAs (tcgen05 cta_group::2, MMA M = 256) works on an item: the rows of a tile as the MMA's N columns (16 to 128 of them, in
// steps of 16, so a tile that is not full costs what its rows do) times 512 weight rows, gate and up rows of 256 neurons or 512 down
// rows, as two accumulators.  Each CTA holds half of the tile's rows and its half of the weight rows, and a chunk of 256 columns
// costs it 77 KB of operands from L2 where a CTA by itself, 128 rows x 256 weight rows, took 108.
// Per CTA: warp 0 the MMA issuer (in the pair's first CTA), warp 1 weights (three stages of 256 columns), warp 2 the items (first CTA),
// warps 4-7 the scale words, 8-11 the tile's rows (ten slots of a (chunk, term)), 12-19 the epilogue (lane = weight row, registers = tile rows).
// The scale words go to tensor memory by tcgen05.st from four warps, one a lane quadrant: tcgen05.cp takes the tensor core ~38 cycles
// each between the MMAs (24 of them beside the 16 MMAs of a chunk: 3360 cycles a chunk instead of 2048), stores from registers run beside it.
// Arrivals on the other CTA's barriers have no cluster-scope release, nor the waits an acquire (with them 6.8 ms instead of 3.2): what they
// announce are bulk copies and tensor-memory stores, which completion, wait::st and the tcgen05 fences order, and cp.async data behind a proxy
// fence.
struct GeoP {
    static constexpr int kBStages = 3, kASlots = 10;
    static constexpr int kBStage = 2 * kBlockF;                       // [codes 0 | scales 0 | codes 1 | scales 1]
    static constexpr int kSFStage = 128 * kSFChunk;                   // the tile's scale bytes of a chunk
    static constexpr int kSlot = 64 * 128;                            // this CTA's half of the tile's rows, one term
    static constexpr int kOffA = kBStages * kBStage, kOffSF = kOffA + kASlots * kSlot, kBars = kOffSF + kBStages * kSFStage;
    static constexpr size_t kSmem = 1024 + (size_t) kBars + 512 + 8 * 64 * sizeof(float2);
    // tensor memory: two accumulators of 128 columns, 16 scale columns a slot, 32 a weight stage
    static constexpr uint32_t kTmemSFB = 256, kTmemSFA = kTmemSFB + 16 * kASlots;
    static constexpr uint32_t kIdesc = (1u << 7) | (1u << 10) | ((uint32_t) (256 >> 4) << 24);      // without N
    static constexpr int kRing = 4;                                   // item numbers on their way
    static_assert(kTmemSFA + 32 * kBStages <= 512 && kBStage % 1024 == 0 && kSlot % 1024 == 0 && kSmem <= 227 * 1024, "geometry");
};
constexpr int kThreadsP = 640;

__device__ __forceinline__ void mma_nvf4_pair(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t accum) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %6, 0;\n"
                 "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%4], [%5], p;\n}\n" ::"r"(d),
                 "l"(ad), "l"(bd), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accum)
                 : "memory");
}
// arrives on the barrier at this place in both CTAs once the MMAs issued so far have finished
__device__ __forceinline__ void commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "h"((uint16_t) 3) : "memory");
}
// arrives on the first CTA's barrier at this place
__device__ __forceinline__ void arrive_first(uint64_t* bar) {
    asm volatile("{\n.reg .b32 m;\nmapa.shared::cluster.u32 m, %0, 0;\nmbarrier.arrive.shared::cluster.b64 _, [m];\n}\n" ::"r"(smem_u32(bar)) : "memory");
}
// a word to the same place in CTA `rank` of the pair, counted in bytes on its barrier at this place
__device__ __forceinline__ void send_word(int* p, int v, uint64_t* bar, uint32_t rank) {
    asm volatile("{\n.reg .b32 m, n;\nmapa.shared::cluster.u32 m, %0, %3;\nmapa.shared::cluster.u32 n, %1, %3;\nmbarrier.arrive.expect_tx.shared::cluster.b64 _, [n], 4;\n"
                 "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.u32 [m], %2, [n];\n}\n" ::"r"(smem_u32(p)), "r"(smem_u32(bar)), "r"(v), "r"(rank)
                 : "memory");
}
__device__ __forceinline__ void pair_sync() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// sixteen columns: the words of w in order, or (tmem_st16t) word i of each vector side by side
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint4 (&w)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n" ::"r"(taddr), "r"(w[0].x),
                 "r"(w[0].y), "r"(w[0].z), "r"(w[0].w), "r"(w[1].x), "r"(w[1].y), "r"(w[1].z), "r"(w[1].w), "r"(w[2].x), "r"(w[2].y), "r"(w[2].z), "r"(w[2].w), "r"(w[3].x),
                 "r"(w[3].y), "r"(w[3].z), "r"(w[3].w)
                 : "memory");
}
__device__ __forceinline__ void tmem_st16t(uint32_t taddr, const uint4 (&w)[4]) {
    const uint4 v[4] = {make_uint4(w[0].x, w[1].x, w[2].x, w[3].x), make_uint4(w[0].y, w[1].y, w[2].y, w[3].y), make_uint4(w[0].z, w[1].z, w[2].z, w[3].z),
                        make_uint4(w[0].w, w[1].w, w[2].w, w[3].w)};
    tmem_st16(taddr, v);
}

// GATHER: the rows come from their own images by cp.async (x rows, which many experts share: laying them out as tile images took 215 us of a
// 16,384-token prompt of 2048 columns); else from tile images by bulk copies (SwiGLU rows: 1.67 ms instead of 1.94 for 73,728 rows of 2048).
template <int MODE, bool GATHER>
__global__ void __launch_bounds__(kThreadsP, 1) prefill_pair_kernel(PrefillFArgs a) {
    using G = GeoP;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t) 1023);
    uint64_t* a_full = reinterpret_cast<uint64_t*>(smem + G::kBars);
    uint64_t* a_empty = a_full + G::kASlots;
    uint64_t* b_full = a_empty + G::kASlots;
    uint64_t* b_empty = b_full + G::kBStages;
    uint64_t* ready = b_empty + G::kBStages;           // [stage]: a chunk's operands landed and scales stored, in both CTAs (the first's counts)
    uint64_t* acc_full = ready + G::kBStages;
    uint64_t* acc_empty = acc_full + 1;                // the first CTA's counts
    uint64_t* item_full = acc_empty + 1;               // [ring]
    uint64_t* item_empty = item_full + G::kRing;       // [ring]: the first CTA's counts
    int* ring = reinterpret_cast<int*>(item_empty + G::kRing);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(ring + G::kRing);
    float2* s_f = reinterpret_cast<float2*>(smem + G::kBars + 512);        // [epilogue warp][64]: its rows' factors (gate, up) or (down, -)

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int rank = (int) (blockIdx.x & 1), pair = (int) (blockIdx.x >> 1), n_pairs = (int) (gridDim.x >> 1);
    const int n_chunk = (int) ((MODE == QMODE_GU ? a.L.n_embd : a.L.n_ff) >> 8);
    const int n_rb = (int) ((MODE == QMODE_GU ? a.L.n_ff : a.L.n_embd) >> 7);      // blocks of 128 weight rows in a matrix, an even number
    const int n_n = MODE == QMODE_GU ? n_rb / 2 : (n_rb + 3) / 4;                    // items a tile
    pdl_wait();
    const TileRec* recs = a.recs;
    const int n_items = *a.n_recs * n_n;
    if (n_items == 0) return;                      // as in most short calls
    const PackedGeom geo = packed_geom(a.L.n_embd, a.L.n_ff);
    // down items of the last blocks may have one accumulator
    auto both = [&](int n) { return MODE == QMODE_GU || 4 * n + 2 < n_rb; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < G::kASlots; ++s) {
            mbar_init(&a_full[s], GATHER ? 128 : 1);
            mbar_init(&a_empty[s], 1);
        }
        for (int s = 0; s < G::kBStages; ++s) {
            mbar_init(&ready[s], 8);               // the scale warps of both CTAs
            mbar_init(&b_full[s], GATHER ? 129 : 2);   // the weight loader's bytes, the row loaders' lanes or bytes (scales)
            mbar_init(&b_empty[s], 1);
        }
        for (int s = 0; s < G::kRing; ++s) {
            mbar_init(&item_full[s], 1);
            mbar_init(&item_empty[s], 1 + 2 * (1 + (GATHER ? 4 : 1) + 4 + 8));        // the roles that read it, in both
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, 16);                  // the epilogue warps of both
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(tmem_slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    pair_sync();                                   // both CTAs' barriers stand before anything arrives on them
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    const uint32_t sbase = smem_u32(smem);
    bool ok = true;

    // Registers: 96 a thread at launch, 48 and 168 from here on: the eight epilogue warps hold an item's 128 values a thread at once.
    // the it-th item of the pair, or -1 after the last (or after a wait that gave up); every role reads them in the same order
    auto read_item = [&](uint32_t it) -> int {
        const uint32_t s = it % G::kRing;
        ok = mbar_wait(&item_full[s], (it / G::kRing) & 1u);
        if (!ok) return -1;
        int item;
        asm volatile("ld.shared.s32 %0, [%1];\n" : "=r"(item) : "r"(smem_u32(ring + s)) : "memory");
        return item;
    };
    auto next_item = [&](uint32_t it) -> int {          // roles of one thread
        const int item = read_item(it);
        arrive_first(&item_empty[it % G::kRing]);
        return item;
    };
    auto next_item_warp = [&](uint32_t it) -> int {
        int item = read_item(it);
        ok = __all_sync(kFull, ok);
        __syncwarp();
        if (lane == 0) arrive_first(&item_empty[it % G::kRing]);
        return ok ? item : -1;
    };
    if (warp >= 12) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 168;\n");
        // ---- epilogue: lane = weight row of both accumulators, registers = tile rows, the first or second 64 of them.  A warp may only
        // read lanes 32 (warp % 4) .. + 31.  All values go to registers first, so the accumulators are back with the tensor core before
        // any of them is worked on; a store writes 32 neighbours of one row.
        const int q = warp & 3, half = (warp - 12) >> 2;
        const uint32_t tbase = tmem + ((uint32_t) (q * 32) << 16) + 64u * half;
        float2* f = s_f + (warp - 12) * 64;
        for (uint32_t ti = 0;; ++ti) {
            const int item = next_item_warp(ti);
            if (item < 0) break;
            const int tile = item / n_n, n = item - tile * n_n;
            const TileRec r = recs[tile];
            const bool two = both(n);
            const int live = r.rows - 64 * half;                     // of this warp's 64 rows
            __syncwarp();
            for (int j = lane; j < min(live, 64); j += 32) {
                const int row = r.row0 + 64 * half + j;
                const float* tail = reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(r.blob) + geo.tail);
                const float iv = a.inv[MODE == QMODE_GU ? a.src[row] : row];
                f[j] = MODE == QMODE_GU ? make_float2(tail[0] * iv, tail[1] * iv) : make_float2(tail[2] * iv, 0.f);
            }
            __syncwarp();
            ok = __all_sync(kFull, mbar_wait(acc_full, ti & 1u));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            uint32_t v0[2][32], v1[2][32];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (live > 32 * i) {
                    tmem_ld32(tbase + 32u * i, v0[i]);
                    if (two) tmem_ld32(tbase + 128u + 32u * i, v1[i]);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) arrive_first(acc_empty);
            if (MODE == QMODE_GU) {
                float* p = a.h + (size_t) (r.row0 + 64 * half) * a.L.n_ff + (size_t) n * 256 + rank * 128 + q * 32 + lane;
                auto store = [&](auto form) {
#pragma unroll
                    for (int i = 0; i < 2; ++i)
#pragma unroll
                        for (int j = 0; j < 32; j += 8) {          // eight at a time, so that their latencies overlap
                            if (32 * i + j >= live) break;
                            float o[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e) {
                                const float2 s = f[32 * i + j + e];
                                o[e] = swiglu_as<decltype(form)::value>(__uint_as_float(v0[i][j + e]) * s.x, __uint_as_float(v1[i][j + e]) * s.y, a.L);
                            }
#pragma unroll
                            for (int e = 0; e < 8; ++e)
                                if (32 * i + j + e < live) p[(size_t) (32 * i + j + e) * a.L.n_ff] = o[e];
                        }
                };
                const int form = swiglu_form(a.L);
                if (form == SWIGLU_PLAIN) store(std::integral_constant<int, SWIGLU_PLAIN>{});
                else if (form == SWIGLU_LIMIT) store(std::integral_constant<int, SWIGLU_LIMIT>{});
                else store(std::integral_constant<int, SWIGLU_CAP>{});
            } else {
                float* p = a.dm + (size_t) (r.row0 + 64 * half) * a.L.n_embd + (size_t) n * 512 + rank * 128 + q * 32 + lane;
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        if (32 * i + j >= live) break;
                        const float s = f[32 * i + j].x;
                        p[0] = __uint_as_float(v0[i][j]) * s;
                        if (two) p[256] = __uint_as_float(v1[i][j]) * s;
                        p += a.L.n_embd;
                    }
            }
        }
        if (!ok && lane == 0) atomicOr(a.status, 1);
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 48;\n");
        if (warp == 0) {
            // ---- MMA issuer
            if (rank == 0 && elect_one()) {
                uint32_t kb = 0, ka = 0;
                for (uint32_t ti = 0; ok; ++ti) {
                    const int item = next_item(ti);
                    if (item < 0) break;
                    const int tile = item / n_n, n = item - tile * n_n;
                    const uint32_t idesc = G::kIdesc | ((uint32_t) ((recs[tile].rows + 15) >> 4) << 18);
                    const bool two = both(n);
                    ok = mbar_wait(acc_empty, (ti & 1u) ^ 1u);
                    if (!ok) break;
                    for (int c = 0; c < n_chunk && ok; ++c, ++kb) {
                        const uint32_t sb = kb % G::kBStages, bst = sbase + sb * G::kBStage, tsfa = tmem + G::kTmemSFA + sb * 32;
                        const uint64_t ad0 = smem_desc_sw128(bst), ad1 = smem_desc_sw128(bst + kBlockF);
                        ok = mbar_wait(&ready[sb], (kb / G::kBStages) & 1u);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll 1
                        for (int t = 0; t < kTermsF; ++t, ++ka) {
                            const uint32_t sa = ka % G::kASlots;
                            const uint64_t bd = smem_desc_sw128(sbase + G::kOffA + sa * G::kSlot);
                            const uint32_t tsfb = tmem + G::kTmemSFB + sa * 16;
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const uint32_t accum = (c | t | k) ? 1u : 0u;
                                mma_nvf4_pair(tmem, ad0 + k * kStepCode, bd + k * kStepCode, idesc, tsfa + 4 * k, tsfb + 4 * k, accum);
                                if (two) mma_nvf4_pair(tmem + 128, ad1 + k * kStepCode, bd + k * kStepCode, idesc, tsfa + 16 + 4 * k, tsfb + 4 * k, accum);
                            }
                            commit_pair(&a_empty[sa]);
                        }
                        commit_pair(&b_empty[sb]);
                    }
                    if (!ok) break;
                    commit_pair(acc_full);
                }
                if (!ok) atomicOr(a.status, 1);
            }
        } else if (warp == 1) {
            // ---- weight loader: a stage is two packed blocks
            if (elect_one()) {
                uint32_t kb = 0;
                for (uint32_t ti = 0; ok; ++ti) {
                    const int item = next_item(ti);
                    if (item < 0) break;
                    const int tile = item / n_n, n = item - tile * n_n;
                    const uint8_t* blob = reinterpret_cast<const uint8_t*>(recs[tile].blob);
                    const size_t mat = (size_t) n_chunk * kBlockF;             // a 128-row block over all of K
                    const uint8_t* b0 = MODE == QMODE_GU ? blob + geo.gate + (2 * n + rank) * mat : blob + geo.down + (4 * n + rank) * mat;
                    const uint8_t* b1 = MODE == QMODE_GU ? blob + geo.up + (2 * n + rank) * mat : b0 + 2 * mat;
                    const bool two = both(n);
                    for (int c = 0; c < n_chunk; ++c, ++kb) {
                        const uint32_t s = kb % G::kBStages;
                        ok = mbar_wait(&b_empty[s], ((kb / G::kBStages) & 1u) ^ 1u);
                        if (!ok) break;
                        const uint32_t st = sbase + s * G::kBStage, bar = smem_u32(&b_full[s]);
                        expect_bytes_q(bar, two ? 2 * kBlockF : kBlockF);
                        bulk_copy_q(st, b0 + (size_t) c * kBlockF, kBlockF, bar);
                        if (two) bulk_copy_q(st + kBlockF, b1 + (size_t) c * kBlockF, kBlockF, bar);
                    }
                }
                if (!ok) atomicOr(a.status, 1);
            }
        } else if (GATHER && warp >= 8) {
            // ---- row loaders, from the rows' images.  Codes: lane = (16-byte piece c8, row r4 of four) of this CTA's half of the tile's columns,
            // rows r4 + 4 i.  Scales, with a chunk's first term: of the whole tile, four lanes a row, the terms' pieces swizzled so that the warps
            // that read a term of 32 rows meet no bank twice.  Rows past the tile's last are left as they are (a column reaches its own
            // results only).  The barriers count the copies as they land, so ten slots' worth are in flight.
            const uint32_t K = (uint32_t) n_chunk * 256u, term = K / 32, c8 = lane & 7, r4 = lane >> 3;       // image offsets in 16 bytes
            const uint32_t dst0 = r4 * 128 + ((c8 ^ r4) << 4), dst1 = (4 + r4) * 128 + ((c8 ^ (4 + r4)) << 4);
            const uint32_t st = lane & 3, sr = lane >> 2, sdst = sr * kSFChunk + ((st ^ ((sr >> 1) & 3)) << 4);
            const int lw = warp - 8;
            uint32_t issued = 0, kb = 0;
            // arrives once this lane's copies so far have landed, without the lane waiting for it
            auto land = [&](uint64_t* bar) { asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];\n" ::"r"(smem_u32(bar)) : "memory"); };
            for (uint32_t ti = 0; ok; ++ti) {
                const int item = next_item_warp(ti);
                if (item < 0) break;
                const TileRec r = recs[item / n_n];
                auto image_row = [&](int row) { return (uint32_t) (MODE == QMODE_GU ? a.src[r.row0 + row] : r.row0 + row); };
                const int per = (r.rows + 15) >> 4, row0 = rank * per * 8, live = (min(r.rows - row0, per * 8) - (int) r4 + 3) >> 2;
                uint32_t off[4], soff[4];          // groups 4 lw .. + 3 of the sixteen of each kind
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    off[i] = image_row(min(row0 + 4 * (4 * lw + i) + (int) r4, r.rows - 1)) * (kTermsF * term) + c8;
                    soff[i] = image_row(min(8 * (4 * lw + i) + (int) sr, r.rows - 1)) * (K / 64) + st;
                }
                for (int c = 0; c < n_chunk && ok; ++c, ++kb)
#pragma unroll 1
                    for (int t = 0; t < kTermsF; ++t) {
                        const uint32_t s = issued % G::kASlots, sb = kb % G::kBStages;
                        ok = mbar_wait(&a_empty[s], ((issued / G::kASlots) & 1u) ^ 1u);
                        if (t == 0) ok = ok && mbar_wait(&b_empty[sb], ((kb / G::kBStages) & 1u) ^ 1u);
                        ok = __all_sync(kFull, ok);
                        if (!ok) break;
                        const uint32_t slot = sbase + (uint32_t) (G::kOffA + s * G::kSlot);
                        const uint8_t* g = a.img + (size_t) (t * term + c * 8) * 16;
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (4 * lw + i < live)
                                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(slot + (uint32_t) ((2 * lw + (i >> 1)) * 1024) + ((i & 1) ? dst1 : dst0)), "l"(g + (size_t) off[i] * 16) : "memory");
                        if (t == 0) {
                            const uint32_t sf = sbase + (uint32_t) (G::kOffSF + sb * G::kSFStage) + sdst;
                            const uint8_t* gs = a.sfs + (size_t) c * kSFChunk;
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                if (8 * (4 * lw + i) + (int) sr < r.rows)
                                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sf + (uint32_t) ((4 * lw + i) * 8 * kSFChunk)), "l"(gs + (size_t) soff[i] * 16) : "memory");
                        }
                        if (t == 0) land(&b_full[sb]);
                        land(&a_full[s]);
                        ++issued;
                    }
            }
            asm volatile("cp.async.wait_all;\n" ::: "memory");
            if (!ok && lane == 0) atomicOr(a.status, 1);
        } else if (!GATHER && warp >= 8) {
            // ---- row loader, from the tile images: the scale words of the whole tile and this CTA's half of its columns, as far as there are rows
            if (warp == 8 && elect_one()) {
                uint32_t ka = 0, kb = 0;
                for (uint32_t ti = 0; ok; ++ti) {
                    const int item = next_item(ti);
                    if (item < 0) break;
                    const TileRec r = recs[item / n_n];
                    const uint32_t bytes = (uint32_t) tile_units(r.rows) * 1024u, atoms = (uint32_t) (r.rows + 7) >> 3, per = (uint32_t) (r.rows + 15) >> 4;
                    const uint32_t off = kSFQ + (rank ? per * 1024u : 0u), mine = (rank ? atoms - per : per) * 1024u;
                    const uint8_t* g = a.img + image_block(r, n_chunk, 0, 0);
                    for (int c = 0; c < n_chunk && ok; ++c, ++kb) {
                        const uint32_t sb = kb % G::kBStages, sbar = smem_u32(&b_full[sb]);
#pragma unroll 1
                        for (int t = 0; t < kTermsF; ++t, ++ka, g += bytes) {
                            const uint32_t s = ka % G::kASlots;
                            ok = mbar_wait(&a_empty[s], ((ka / G::kASlots) & 1u) ^ 1u);
                            if (t == 0) ok = ok && mbar_wait(&b_empty[sb], ((kb / G::kBStages) & 1u) ^ 1u);
                            if (!ok) break;
                            if (t == 0) expect_bytes_q(sbar, kTermsF * kSFQ);
                            bulk_copy_q(sbase + (uint32_t) (G::kOffSF + sb * G::kSFStage + t * kSFQ), g, kSFQ, sbar);
                            const uint32_t bar = smem_u32(&a_full[s]);
                            expect_bytes_q(bar, mine);
                            if (mine) bulk_copy_q(sbase + (uint32_t) (G::kOffA + s * G::kSlot), g + off, mine, bar);
                        }
                    }
                }
                if (!ok) atomicOr(a.status, 1);
            }
        } else if (warp == 2) {
            // ---- items: the pair's own number first, then from the launch's counter, a few ahead of the roles.  Tiles differ in their rows, so
            // items dealt in turn would leave the fullest pair 4 to 20 % behind the average.
            if (rank == 0 && elect_one()) {
                int item = pair;
                for (uint32_t it = 0; ok; ++it) {
                    const uint32_t s = it % G::kRing;
                    ok = mbar_wait(&item_empty[s], ((it / G::kRing) & 1u) ^ 1u);
                    if (!ok) break;
                    const int v = item < n_items ? item : -1;
                    send_word(ring + s, v, &item_full[s], 1);
                    send_word(ring + s, v, &item_full[s], 0);
                    if (v < 0) break;
                    item = n_pairs + atomicAdd(a.counter, 1);
                }
                if (!ok) atomicOr(a.status, 1);
            }
        } else if (warp >= 4) {
            // ---- scale words, shared -> tensor memory: lane l of each quadrant takes the words of rows l, l + 32, l + 64, l + 96 of a K-step
            const uint32_t quad = (uint32_t) ((warp & 3) * 32) << 16;
            auto fetch = [&](uint32_t from, uint32_t step, uint4 (&w)[4]) {
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(w[i].x), "=r"(w[i].y), "=r"(w[i].z), "=r"(w[i].w) : "r"(from + i * step) : "memory");
            };
            uint32_t kb = 0, ka = 0;
            for (uint32_t ti = 0; ok; ++ti) {
                const int item = next_item_warp(ti);
                if (item < 0) break;
                const bool two = both(item % n_n);
                for (int c = 0; c < n_chunk; ++c, ++kb) {
                    // a chunk at a time: one wait for the stores, one arrival (a slot at a time the loop's latency held the tensor core back)
                    const uint32_t sb = kb % G::kBStages, bst = sbase + sb * G::kBStage + kATileQ + lane * 16, tsfa = tmem + quad + G::kTmemSFA + sb * 32;
                    const uint32_t sf = sbase + (uint32_t) (G::kOffSF + sb * G::kSFStage) + lane * (GATHER ? kSFChunk : 16);
                    ok = __all_sync(kFull, mbar_wait(&b_full[sb], (kb / G::kBStages) & 1u));
                    if (!ok) break;
                    __syncwarp();
                    uint4 w0[4], w1[4];
                    fetch(bst, 512, w0);                       // weights: a K-step's words of four rows a lane lie together
                    if (two) fetch(bst + kBlockF, 512, w1);
                    tmem_st16(tsfa, w0);
                    if (two) tmem_st16(tsfa + 16, w1);
#pragma unroll
                    for (int t = 0; t < kTermsF; t += 2, ka += 2) {
                        const uint32_t s0 = ka % G::kASlots, s1 = (ka + 1) % G::kASlots;
                        ok = ok && mbar_wait(&a_full[s0], (ka / G::kASlots) & 1u) && mbar_wait(&a_full[s1], ((ka + 1) / G::kASlots) & 1u);
                        __syncwarp();
                        if (GATHER) {                          // a row's words of four K-steps lie together
                            fetch(sf + ((t ^ ((lane >> 1) & 3)) << 4), 32 * kSFChunk, w0);
                            fetch(sf + (((t + 1) ^ ((lane >> 1) & 3)) << 4), 32 * kSFChunk, w1);
                            tmem_st16t(tmem + quad + G::kTmemSFB + s0 * 16, w0);
                            tmem_st16t(tmem + quad + G::kTmemSFB + s1 * 16, w1);
                        } else {
                            fetch(sf + t * kSFQ, 512, w0);
                            fetch(sf + (t + 1) * kSFQ, 512, w1);
                            tmem_st16(tmem + quad + G::kTmemSFB + s0 * 16, w0);
                            tmem_st16(tmem + quad + G::kTmemSFB + s1 * 16, w1);
                        }
                    }
                    ok = __all_sync(kFull, ok);
                    if (!ok) break;
                    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
                    if (GATHER) asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");        // the rows' codes, which cp.async wrote, to the tensor core
                    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                    __syncwarp();
                    if (lane == 0) arrive_first(&ready[sb]);
                }
            }
            if (!ok && lane == 0) atomicOr(a.status, 1);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    pair_sync();                                   // the other CTA arrives on this one's barriers no more
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
    }
}

template <int MODE, bool GATHER>
int32_t launch_pair(const PrefillFArgs& a, cudaStream_t st) {
    static std::atomic<bool> configured[64];   // per device; threads of different devices call concurrently
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return (int32_t) cudaErrorInvalidDevice;
    if (!configured[dev].load(std::memory_order_acquire)) {
        const cudaError_t e = cudaFuncSetAttribute(prefill_pair_kernel<MODE, GATHER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) GeoP::kSmem);
        if (e != cudaSuccess) return (int32_t) e;
        configured[dev].store(true, std::memory_order_release);
    }
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned) (sm_count() / 2 * 2));
    cfg.blockDim = dim3(kThreadsP);
    cfg.dynamicSmemBytes = GeoP::kSmem;
    cfg.stream = st;
    cfg.attrs = at;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.numAttrs = 2;
    (void) cudaLaunchKernelEx(&cfg, prefill_pair_kernel<MODE, GATHER>, a);
    return launch_status();
}

size_t al256q(size_t v) { return (v + 255) & ~(size_t) 255; }

}  // namespace
}  // namespace bsx

using namespace bsx;

// Rows an expert, on average over the call, up to which the decode stream takes it: from there on its second and third passes over an expert's
// weights outweigh what tiles cost beside the rows.  Expert stage, rows dealt at random, stream against tiles, us: 2048 x 512 with 513 experts
// at 26 rows an expert 279 : 298, 28 286 : 305, 30 301 : 316, 32 320 : 320; 5120 x 2304 with 385 at 26 1828 : 1948, 28 1920 : 1974, 30
// 1999 : 1985, 32 2109 : 2028; 7168 x 2048 with 257 at 26 1503 : 1599, 28 1556 : 1613, 30 1650 : 1620.  An n_ff of 256 leaves a down item one
// chunk, which its epilogue outlasts: 2048 x 256 with 513 experts at 30 202 : 232, 38 248 : 255; 4096 x 256 at 34 373 : 373; 7168 x 256 with 257 at
// 38 350 : 358, 42 372 : 366.
static int64_t short_rows(const bsx_expert_layout& L) { return L.n_ff == 256 ? 38 : 29; }
// Rows an expert from which the SwiGLU rows are laid out as tile images: these hold up to 23 rows more a tile than there are.
constexpr int64_t kTileImageRows = 48;

// Rows of up to 1025 experts make at most this many tiles.
static int64_t prefill_cap_tiles(int64_t cap_rows, int64_t n_expert) { return std::min(cap_rows, cap_rows / 128 + std::min<int64_t>(n_expert, 1025)); }

// Where a call's buffers lie in its scratch, and the route that its numbers choose.
struct PrefillCarve {
    bool stream, h_tiles;              // few rows an expert: the decode stream; many: tile images of the SwiGLU rows
    int64_t cap_recs, cap_items, cap_units;
    size_t xcodes, xsf, xinv, h, hcodes, hsf, hinv, recs, n_recs, items, n_items, bytes;
};
// n_held of the n_expert experts have blobs here.
static PrefillCarve prefill_carve(const bsx_expert_layout& L, int64_t n_tokens, int64_t cap_rows, int64_t n_expert, int64_t n_held) {
    PrefillCarve c = {};
    const int64_t H = L.n_embd, I = L.n_ff;
    c.stream = cap_rows <= short_rows(L) * n_expert && n_tokens <= 0x7FFFFFFF;
    c.cap_recs = prefill_cap_tiles(cap_rows, n_held);
    c.cap_items = c.stream ? cap_rows / kPassEntries + c.cap_recs : 0;
    if (c.stream) c.cap_recs = std::min(c.cap_recs, cap_rows / (kCrowdedRows + 1) + 1);        // the crowded tiles
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t r = at;
        at += al256q(bytes);
        return r;
    };
    c.xcodes = take((size_t) n_tokens * kTermsF * H / 2);
    c.xsf = take((size_t) n_tokens * kTermsF * H / 16);
    c.xinv = take((size_t) n_tokens * 4);
    c.h = take((size_t) (cap_rows + 128) * I * 4);
    c.h_tiles = cap_rows > kTileImageRows * n_expert;
    c.cap_units = image_units(cap_rows, c.cap_recs);
    if (c.h_tiles) {
        c.hcodes = take((size_t) c.cap_units * 1024 * kTermsF * (I / 256));
    } else {
        c.hcodes = take((size_t) cap_rows * kTermsF * I / 2);
        c.hsf = take((size_t) cap_rows * kTermsF * I / 16);
    }
    c.hinv = take((size_t) (cap_rows + 128) * 4);
    c.recs = take((size_t) c.cap_recs * sizeof(TileRec));
    c.n_recs = take(12);
    c.items = take((size_t) c.cap_items * sizeof(PassRec));
    c.n_items = take(4);
    c.bytes = at;
    return c;
}

extern "C" size_t bsx_experts_prefill_packed_held_scratch_bytes(const bsx_expert_layout* L, int64_t n_tokens, int64_t cap_rows, int32_t n_expert, int32_t n_held) {
    if (!L || n_tokens < 0 || cap_rows < 0 || n_expert < 1 || n_held < 0 || n_held > n_expert || !bsx_expert_packed_bytes(L)) return 0;
    // A caller may size its scratch by its largest call, and the longest short one can need a little more than the next: its pass records.
    return std::max(prefill_carve(*L, n_tokens, cap_rows, n_expert, n_held).bytes,
                    prefill_carve(*L, n_tokens, std::min(cap_rows, short_rows(*L) * n_expert), n_expert, n_held).bytes);
}

// the most that any number of experts needs: of each route, for the largest number that takes it
extern "C" size_t bsx_experts_prefill_packed_scratch_bytes(const bsx_expert_layout* L, int64_t n_tokens, int64_t cap_rows) {
    if (!L || n_tokens < 0 || cap_rows < 0 || !bsx_expert_packed_bytes(L)) return 0;
    const int64_t few = short_rows(*L), number[3] = {std::max<int64_t>(1025, (cap_rows + few - 1) / few), (cap_rows - 1) / few, (cap_rows - 1) / kTileImageRows};
    size_t most = 0;
    for (int64_t n : number)
        if (n >= 1) most = std::max(most, prefill_carve(*L, n_tokens, cap_rows, n, n).bytes);
    return most;
}

extern "C" int32_t bsx_experts_prefill_packed_held(const bsx_expert_layout* layout, const unsigned long long* blob_table, const int32_t* off,
                                                   const int32_t* src, const int32_t* tiles, const int32_t* n_tiles, int64_t cap_tiles, int64_t cap_rows,
                                                   const void* x, int32_t x_kind, int64_t n_tokens, int32_t n_expert, int32_t n_held, void* scratch, float* dm,
                                                   int32_t* status, void* stream) {
    if (!stream) return BSX_E_STREAM;
    if (!layout || !blob_table || !off || !src || !tiles || !n_tiles || !aligned(x, 16) || !aligned(scratch, 256) || !aligned(dm, 16) || !status)
        return BSX_E_POINTER;
    if (!bsx_expert_packed_bytes(layout)) return BSX_E_TYPE;
    if (x_kind != BSX_X_F32 && x_kind != BSX_X_BF16) return BSX_E_GEOMETRY;
    if (cap_tiles < 0 || cap_rows < 0 || n_tokens < 0 || n_expert < 1 || n_held < 0 || n_held > n_expert) return BSX_E_GEOMETRY;
    if (cap_tiles == 0 || n_tokens == 0 || cap_rows == 0 || n_held == 0) return BSX_OK;
    if (cap_tiles > cap_rows / 128 + 1025) return BSX_E_LIMIT;      // more tiles than rows / 128 + experts can make
    const bsx_expert_layout& L = *layout;
    const cudaStream_t st = (cudaStream_t) stream;
    const int64_t H = L.n_embd, I = L.n_ff;
    const PrefillCarve c = prefill_carve(L, n_tokens, cap_rows, n_expert, n_held);
    uint8_t* base = static_cast<uint8_t*>(scratch);
    uint8_t *xcodes = base + c.xcodes, *xsf = base + c.xsf, *hcodes = base + c.hcodes, *hsf = base + c.hsf;
    float *xinv = reinterpret_cast<float*>(base + c.xinv), *h = reinterpret_cast<float*>(base + c.h), *hinv = reinterpret_cast<float*>(base + c.hinv);
    RecordArgs ra;
    ra.tiles = tiles;
    ra.n_tiles = n_tiles;
    ra.off = off;
    ra.blob_table = blob_table;
    ra.cap_tiles = cap_tiles;
    ra.recs = reinterpret_cast<TileRec*>(base + c.recs);
    ra.cap_recs = c.cap_recs;
    ra.n_recs = reinterpret_cast<int32_t*>(base + c.n_recs);
    ra.cap_units = c.cap_units;
    ra.items = c.stream ? reinterpret_cast<PassRec*>(base + c.items) : nullptr;
    ra.n_items = c.stream ? reinterpret_cast<int*>(base + c.n_items) : nullptr;
    ra.cap_items = c.cap_items;
    ra.pass_entries = cap_rows > kPassEntries / 2 * n_expert ? 2 * kPassEntries : kPassEntries;
    ra.tile_items = (int) (I / 128);
    ra.sm_count = sm_count();
    ra.status = status;
    PrefillFArgs a;
    a.L = L;
    a.recs = ra.recs;
    a.n_recs = ra.n_recs;
    a.src = src;
    a.h = h;
    a.dm = dm;
    a.status = status;
    ExpertArgs e;
    e.L = L;
    e.grp_ptr = nullptr;
    e.grp_start = nullptr;
    e.n_groups = nullptr;
    e.ent_dst = nullptr;
    e.ent_tok = src;
    e.cap_groups = n_expert;
    e.cap_entries = cap_rows;
    e.x = x;
    e.x_kind = x_kind;
    e.h = h;
    e.out = dm;
    e.out_kind = BSX_OUT_F32;
    e.n_x_rows = (int32_t) n_tokens;
    e.grid = nullptr;
    // Few rows an expert: the rows go through the decode stream (experts_nvf4.cu: passes of 8 or 16 rows, bound by the weights), crowded tiles
    // aside (tile_records_kernel), which in most calls there are none of: their kernels then return at once.  Else every tile is a tile.
    PdlScope pdl(true, 1);      // the first kernel follows the caller's work
    launch_k(tile_records_kernel, dim3(1), dim3(1024), 0, st, ra);
    packed_x_images(x, x_kind, n_tokens, H, xcodes, xsf, xinv, st);
    a.img = xcodes;
    a.sfs = xsf;
    a.inv = xinv;
    a.counter = ra.n_recs + 1;
    int32_t rc = launch_pair<QMODE_GU, true>(a, st);
    if (rc == BSX_OK && c.stream) rc = packed_pass_product(false, e, ra.items, ra.n_items, ra.pass_entries, xcodes, xsf, xinv, status, st);
    if (rc != BSX_OK) return rc;
    if (!c.h_tiles) packed_listed_images(h, ra.items, ra.n_items, ra.pass_entries, ra.recs, ra.n_recs, I, hcodes, hsf, hinv, st);
    else if (I <= 512) launch_k(h_images_kernel<1>, dim3((unsigned) (c.cap_recs * 16)), dim3(256), 0, st, a.recs, a.n_recs, h, I, hcodes, hinv);
    else launch_k(h_images_kernel<0>, dim3((unsigned) (c.cap_recs * 16)), dim3(256), 0, st, a.recs, a.n_recs, h, I, hcodes, hinv);
    a.img = hcodes;
    a.sfs = hsf;
    a.inv = hinv;
    a.counter = ra.n_recs + 2;
    rc = c.h_tiles ? launch_pair<QMODE_DOWN, false>(a, st) : launch_pair<QMODE_DOWN, true>(a, st);
    if (rc == BSX_OK && c.stream) rc = packed_pass_product(true, e, ra.items, ra.n_items, ra.pass_entries, hcodes, hsf, hinv, status, st);
    return rc;
}

extern "C" int32_t bsx_experts_prefill_packed(const bsx_expert_layout* layout, const unsigned long long* blob_table, const int32_t* off,
                                              const int32_t* src, const int32_t* tiles, const int32_t* n_tiles, int64_t cap_tiles, int64_t cap_rows,
                                              const void* x, int32_t x_kind, int64_t n_tokens, int32_t n_expert, void* scratch, float* dm, int32_t* status,
                                              void* stream) {
    return bsx_experts_prefill_packed_held(layout, blob_table, off, src, tiles, n_tiles, cap_tiles, cap_rows, x, x_kind, n_tokens, n_expert, n_expert, scratch, dm,
                                           status, stream);
}
