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
// Persistent CTAs, one per SM, static round-robin over work items (128-row tile of one expert x 256 weight rows: gate/up 128 gate
// rows and their 128 up rows, down 256 rows; one accumulator of 256 columns).  Every operand is a bulk copy: the rows of a tile are
// laid out beforehand as the images a stage holds (tile_images_kernel for x, h_images_kernel for the SwiGLU rows).  Warp 0: per
// 64-column K-step the scale copies (tcgen05.cp shared -> tensor memory) and one MMA a term (M = 128 rows); warp 1: weights, two
// stages of 256 columns; warp 2: activations, a slot a (chunk, term), eight of them, so that a slot is refilled as soon as its four
// MMAs have read it; warps 4-11: epilogue (thread = TMEM lane = row).  Every wait is time-bounded with a status word.
// Bound: operands from L2, 108 KB a (tile, 256 rows, 256 columns) against 2048 tensor-core cycles; the copies alone run at 10.6 TB/s
// over the chip.  Measured, gate/up product of the 7168 x 2048 layer at 8192 tokens (256 experts + the shared one): 4.88 ms with
// rows gathered by cp.async and MMAs issued under `lane == 0`, 4.59 with bulk copies, 3.52 with the issue under elect.sync too
// (tc5.cuh); its down product 3.80 -> 2.33 (256 instead of 128 rows an item) -> 1.87.
// With n_ff <= 512 the down product runs as prefill_down_resident_kernel instead (the tile's rows stay in shared memory).
#include <algorithm>
#include <atomic>
#include <cuda_fp16.h>

#include "common.cuh"
#include "experts.cuh"
#include "nvf4.cuh"
#include "pdl.cuh"
#include "plan.cuh"
#include "tc5.cuh"

namespace bsx {

void packed_x_images(const void* x, int kind, int64_t rows, int64_t K, uint8_t* codes, uint8_t* sfs, float* inv, cudaStream_t st);
void packed_listed_images(const float* h, const PassRec* items, const int* n_items, int pass_entries, const TileRec* recs, const int32_t* slab, int64_t K, uint8_t* codes,
                          uint8_t* sfs, float* inv, cudaStream_t st);
int32_t packed_pass_product(bool down, const ExpertArgs& a, const PassRec* items, const int* n_items, int pass_entries, const uint8_t* codes, const uint8_t* sfs,
                            const float* inv, int32_t* status, cudaStream_t st);

namespace {

constexpr int kThreadsQ = 32 * 12;
constexpr int kATileQ = 128 * 128;                 // code tile of 128 rows x 256 columns
constexpr int kSFQ = 4 * 512;                      // its scale words: four K-steps of 32 lanes x 4 words
constexpr int kSlotQ = kSFQ + kATileQ;             // an activation slot: [scale words | codes], 18,432 bytes = a packed block's size
constexpr int kBStages = 2, kASlots = kBStages * kTermsF;
enum { QMODE_GU = 0, QMODE_DOWN = 1 };

struct GeoQ {
    // shared memory: kBStages x [codes 0 | codes 1 | scales 0 | scales 1], then kASlots x [scales | codes], then the barriers
    static constexpr int kBStage = 2 * kBlockF;
    static constexpr int kOffA = kBStages * kBStage;
    static constexpr int kBars = kOffA + kASlots * kSlotQ;
    static constexpr size_t kSmem = 1024 + (size_t) kBars + 256;
    // tensor memory: one accumulator of 256 columns, 16 scale columns per activation slot, 32 per weight stage
    static constexpr uint32_t kTmemSFA = 256, kTmemSFB = kTmemSFA + 16 * kASlots;
    static constexpr uint32_t kIdesc = (1u << 7) | (1u << 10) | ((uint32_t) (256 >> 3) << 17) | ((uint32_t) (128 >> 4) << 24);
};

// Tile images.  The activation rows a tile multiplies lie in dispatch order, in the form a stage has in shared memory: for each
// (chunk of 256 columns, FP4 term) one run of [2 KB scale words, as tcgen05.cp reads them for 128 rows | 1 KB per eight rows of
// codes, 128-byte swizzled], so that a stage of a tile is one bulk copy and a tile with few rows is a short one.  A tile takes
// `units` = ceil(rows / 8) + 2 KB per (chunk, term); rows and scale words past its last row are never written (each only
// reaches its own accumulator row, which is not stored).
constexpr int kMaxUnits = 128 / 8 + 2;
__host__ __device__ __forceinline__ int tile_units(int rows) { return (rows + 7) / 8 + 2; }
__device__ __forceinline__ size_t image_block(const TileRec& r, int n_chunk, int c, int t) {
    return ((size_t) r.base * n_chunk * kTermsF + (size_t) (c * kTermsF + t) * tile_units(r.rows)) * 1024;
}

// units that cap_rows rows in cap_tiles tiles can take
__host__ __device__ inline int64_t image_units(int64_t cap_rows, int64_t cap_tiles) { return cap_rows / 8 + 3 * cap_tiles; }

// The tile list without the tiles of experts held elsewhere, cut into slabs of slab_units units: slab s is the tiles
// slab_first[s] .. slab_first[s + 1] - 1, those whose units before them are s slabs' worth, so a slab's images end at most one tile
// past slab_units.  One block; a scan carries units and places together.  Tiles that overlap (no dispatch makes them) and exceed the
// room are left out and set the status word.
// items (optional, a short call): the rows become passes of up to pass_entries rows for the decode stream instead.  But a call that is
// short by its average may still send most rows to a few experts, and the stream reads an expert's weights once a pass: tiles of more
// than kCrowdedRows rows then are one slab of tiles, provided the passes they save outweigh what the tile kernels take in the
// whole.  A tile costs the chip about as much as three passes (5120 x 2304 with 27 rows an expert: 7.0 and 2.4 us), and the tile
// kernels come in rounds of sm_count items, of which a call pays one more than it fills (launches, the last item's latency).
constexpr int kCrowdedRows = 64;
struct RecordArgs {
    const int32_t *tiles, *n_tiles, *off;
    const unsigned long long* blob_table;
    int64_t cap_tiles;
    TileRec* recs;
    int64_t cap_recs;
    int32_t* slab_first;
    int n_slabs;
    int64_t slab_units;
    PassRec* items;
    int* n_items;
    int64_t cap_items;
    int pass_entries, tile_items, sm_count;      // tile_items: items of a tile's gate/up product
    int32_t* status;
};
__global__ void __launch_bounds__(1024) tile_records_kernel(RecordArgs a) {
    __shared__ unsigned long long sh[32];
    constexpr unsigned long long kLow = (1ull << 36) - 1;               // units or passes | tiles << 36
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
        const int passes = a.items && !tile ? (r.rows + a.pass_entries - 1) / a.pass_entries : 0, u = tile ? tile_units(r.rows) : 0;
        unsigned long long total = 0;
        const unsigned long long before =
            block_excl_sum<unsigned long long>((unsigned long long) (a.items ? passes : u) | ((unsigned long long) tile << 36), &total, sh);
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
        const int64_t slab = a.items ? 0 : at / a.slab_units, next = a.items ? 0 : (at + u) / a.slab_units;
        r.base = at - slab * a.slab_units;
        if (place < a.cap_recs) a.recs[place] = r;
        if (next > slab && next <= a.n_slabs) a.slab_first[next] = (int) min(place + 1, a.cap_recs);   // u <= slab_units: at most one slab begins here
    }
    if (threadIdx.x == 0) {
        if (placed > a.cap_recs || low > (a.items ? a.cap_items : a.n_slabs * a.slab_units)) atomicOr(a.status, 1);
        if (a.items) *a.n_items = (int) min(low, a.cap_items);
        a.slab_first[0] = 0;
    }
    for (int64_t s = (a.items ? 0 : min(low / a.slab_units, (int64_t) a.n_slabs)) + 1 + threadIdx.x; s <= a.n_slabs; s += 1024)
        a.slab_first[s] = (int) min(placed, a.cap_recs);
}

// The first slab's begin is not read: the image kernels, whose blocks live a few microseconds, need not wait for it before their record.
__device__ __forceinline__ int first_tile(const int32_t* from) { return from ? *from : 0; }

struct PrefillFArgs {
    bsx_expert_layout L;
    const TileRec* recs;                     // every tile of the call
    const int32_t *from, *to;                // the tiles of this launch, *from .. *to - 1 (from: null for 0)
    const int32_t* src;                      // [rows] token of each row
    const uint8_t* img;                      // tile images of this product's A operand; or (GATHER) its rows' images
    const uint8_t* sfs;                      // GATHER: the rows' scales
    const float* inv;
    float* h;                                // [rows + 128][I] fp32 SwiGLU output
    float* dm;                               // [rows][H] fp32
    int32_t* status;
};

__device__ __forceinline__ uint64_t sf_desc_q(uint32_t addr) {   // 32 rows x 16 bytes, 8-row groups 128 bytes apart, no swizzle
    return (uint64_t) ((addr & 0x3FFFFu) >> 4) | ((uint64_t) (128 >> 4) << 16) | ((uint64_t) (128 >> 4) << 32) | ((uint64_t) 1 << 46);
}
__device__ __forceinline__ void sf_copy_q(uint32_t tmem_addr, uint64_t desc) {
    asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;\n" ::"r"(tmem_addr), "l"(desc) : "memory");
}
__device__ __forceinline__ void mma_nvf4_q(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t sfa, uint32_t sfb, uint32_t accum) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %6, 0;\n"
                 "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.scale_vec::4X [%0], %1, %2, %3, [%4], [%5], p;\n}\n" ::"r"(d),
                 "l"(ad), "l"(bd), "r"(idesc), "r"(sfa), "r"(sfb), "r"(accum)
                 : "memory");
}
__device__ __forceinline__ void bulk_copy_q(uint32_t dst, const uint8_t* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void expect_bytes_q(uint32_t bar, uint32_t bytes) {
    asm volatile("{\n.reg .b64 t;\nmbarrier.arrive.expect_tx.shared::cta.b64 t, [%0], %1;\n}\n" ::"r"(bar), "r"(bytes) : "memory");
}
// descriptors count addresses in 16 bytes: a K-step further is 32 bytes of codes, 512 of scale words
constexpr uint64_t kStepCode = 2, kStepSF = 32;
// eight consecutive floats of one row.  A thread of the epilogue owns a row, so a store instruction touches 32 rows: 32 bytes each
// fill a sector, 16 bytes (rows whose base is only 16-byte aligned) would write every sector in two halves.
__device__ __forceinline__ void store8_q(float* p, const float (&v)[8], bool wide) {
    if (wide) {
        asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]),
                     "f"(v[6]), "f"(v[7])
                     : "memory");
    } else {
        reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
    }
}

// 32 consecutive floats of each lane's row to memory.  A lane owns a row, so storing straight from the registers would touch 32
// lines an instruction; a 4 x 4 transposition among neighbouring lanes makes four lanes hold one row's 128 bytes, eight lines an
// instruction (the resident down product of 180,224 rows x 2048: 495 -> 458 us).  base: column 0 of the row of lane 0 of the
// warp; rows beyond `live` are not stored.  wide: 32-byte aligned rows.
__device__ __forceinline__ void store_rows32_q(float* base, size_t pitch, int live, int lane, float (&v)[32], bool wide) {
#pragma unroll
    for (int s = 1; s <= 2; s <<= 1)
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (u & s) continue;
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                float& lo = v[8 * u + e];
                float& hi = v[8 * (u | s) + e];
                const float r = __shfl_xor_sync(kFull, (lane & s) ? lo : hi, s);
                if (lane & s) lo = r;
                else hi = r;
            }
        }
    const int row = lane & ~3;
    float* p = base + (size_t) row * pitch + (lane & 3) * 8;
#pragma unroll
    for (int i = 0; i < 4; ++i, p += pitch) {
        if (row + i >= live) break;
        if (wide) {
            asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"l"(p), "f"(v[8 * i]), "f"(v[8 * i + 1]), "f"(v[8 * i + 2]),
                         "f"(v[8 * i + 3]), "f"(v[8 * i + 4]), "f"(v[8 * i + 5]), "f"(v[8 * i + 6]), "f"(v[8 * i + 7])
                         : "memory");
        } else {
            reinterpret_cast<float4*>(p)[0] = make_float4(v[8 * i], v[8 * i + 1], v[8 * i + 2], v[8 * i + 3]);
            reinterpret_cast<float4*>(p)[1] = make_float4(v[8 * i + 4], v[8 * i + 5], v[8 * i + 6], v[8 * i + 7]);
        }
    }
}

// rows of x (fp32 or bf16) -> FP4 terms, one image row per token: codes [token][term][H / 2], scales [token][term][H / 16]
template <int TPR>
__global__ void __launch_bounds__(256) prefill_images_kernel(const void* __restrict__ src, int kind, int64_t n, int64_t K, uint8_t* __restrict__ codes,
                                                              uint8_t* __restrict__ sfs, float* __restrict__ inv) {
    __shared__ float shf[8];
    const int64_t i = (int64_t) blockIdx.x * (256 / TPR) + threadIdx.x / TPR;
    fp4_image_row<TPR>(src, kind, i < n ? i : 0, K, i < n, (int) i, codes, sfs, inv, shf);
}

// token images -> tile images of the gate/up product.  Block = one (tile, chunk): every row's four 128-byte code runs move in
// 16-byte pieces (eight lanes a run), the scale words are transposed through shared memory.  Bound: HBM writes of 2.25 bytes a
// value (180,224 rows x 2048: 830 MB); the stores are streaming, so that the token images they are read from stay in L2 (247 -> 215 us).
__global__ void __launch_bounds__(256) tile_images_kernel(const TileRec* __restrict__ recs, const int32_t* __restrict__ from, const int32_t* __restrict__ to, int tile0,
                                                          const int32_t* __restrict__ src, const uint8_t* __restrict__ codes, const uint8_t* __restrict__ sfs, int64_t K,
                                                          uint8_t* __restrict__ img) {
    __shared__ __align__(16) uint32_t sf[kTermsF * kSFQ / 4];
    const int tile = first_tile(from) + tile0 + blockIdx.y;
    if (tile >= *to) return;
    const TileRec r = recs[tile];
    const int c = blockIdx.x, n_chunk = gridDim.x;
    uint8_t* out = img + image_block(r, n_chunk, c, 0);
    const size_t term_bytes = (size_t) tile_units(r.rows) * 1024;
    for (int i = threadIdx.x; i < r.rows * kTermsF; i += 256) {        // a row's 16 scale bytes of a term: one word into each K-step's block
        const int row = i >> 2, t = i & 3;
        const uint4 v = *reinterpret_cast<const uint4*>(sfs + ((size_t) src[r.row0 + row] * kTermsF + t) * (size_t) (K >> 4) + (size_t) c * 16);
        uint32_t* d = sf + t * (kSFQ / 4) + (row & 31) * 4 + (row >> 5);
        d[0] = v.x;
        d[128] = v.y;
        d[256] = v.z;
        d[384] = v.w;
    }
    const int p = threadIdx.x & 7;
    for (int row0 = threadIdx.x >> 5; row0 < r.rows; row0 += 32) {     // a warp: a row's four terms, four rows in flight
        const int t = (threadIdx.x >> 3) & 3;
        uint4 v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int row = min(row0 + 8 * j, r.rows - 1);
            v[j] = *reinterpret_cast<const uint4*>(codes + ((size_t) src[r.row0 + row] * kTermsF + t) * (size_t) (K >> 1) + (size_t) c * 128 + p * 16);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int row = row0 + 8 * j;
            if (row < r.rows) __stcs(reinterpret_cast<uint4*>(out + t * term_bytes + kSFQ + (row >> 3) * 1024 + (row & 7) * 128 + ((p ^ (row & 7)) << 4)), v[j]);
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kTermsF * kSFQ / 16; i += 256) {
        const int t = i / (kSFQ / 16), q = i - t * (kSFQ / 16);
        __stcs(reinterpret_cast<uint4*>(out + t * term_bytes) + q, reinterpret_cast<const uint4*>(sf)[i]);
    }
}

// rows of h (fp32, dispatch order) -> tile images of the down product.  Block = eight rows of a tile, a warp a row: a lane makes
// one sub-block of 16 values at a time, and four lanes' scale bytes make the word tcgen05.cp reads.  NIT = 1: a lane's one sub-block
// stays in registers between the row's maximum and its codes (n_ff <= 512: 205 -> 174 us for 180,224 rows of 512); 0 reads the row
// twice (four sub-blocks in registers were slower there: 274 -> 340 us for 73,728 rows of 2048).
template <int NIT>
__global__ void __launch_bounds__(256) h_images_kernel(const TileRec* __restrict__ recs, const int32_t* __restrict__ from, const int32_t* __restrict__ to, const float* __restrict__ h, int64_t K,
                                                       uint8_t* __restrict__ img, float* __restrict__ inv) {
    const int tile = first_tile(from) + (int) (blockIdx.x >> 4), row = (blockIdx.x & 15) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (tile >= *to) return;
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

// the common start and end of the product kernels: tensor memory for the CTA
__device__ __forceinline__ uint32_t tmem_take_q(uint32_t* slot, int warp) {
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(slot)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    return *slot;
}
__device__ __forceinline__ void tmem_give_q(uint32_t tmem, int warp) {
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// GATHER: the rows come from their own images instead (two warps of cp.async, warps 2 and 3), which takes no room that grows with the
// tiles.  For the crowded tiles of short calls: 1300 rows on nine experts of the 7168 x 2048 layer take 1.43 ms so, 2.03 through the
// stream alone.
template <int MODE, bool GATHER>
__global__ void __launch_bounds__(kThreadsQ, 1) prefill_nvf4_kernel(PrefillFArgs a) {
    using G = GeoQ;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t) 1023);
    uint64_t* a_full = reinterpret_cast<uint64_t*>(smem + G::kBars);
    uint64_t* a_empty = a_full + kASlots;
    uint64_t* b_full = a_empty + kASlots;
    uint64_t* b_empty = b_full + kBStages;
    uint64_t* acc_full = b_empty + kBStages;
    uint64_t* acc_empty = acc_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 1);

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int n_chunk = (int) ((MODE == QMODE_GU ? a.L.n_embd : a.L.n_ff) >> 8);
    const int n_n = (int) (MODE == QMODE_GU ? a.L.n_ff / 128 : a.L.n_embd / 256);   // items per row tile: 128 neurons, or 256 down rows
    if (GATHER) pdl_wait();
    const TileRec* recs = a.recs + first_tile(a.from);
    const int n_items = (*a.to - first_tile(a.from)) * n_n;
    if (GATHER && n_items == 0) return;
    const PackedGeom geo = packed_geom(a.L.n_embd, a.L.n_ff);

    if (threadIdx.x == 0) {
        for (int s = 0; s < kASlots; ++s) {
            mbar_init(&a_full[s], GATHER ? 64 : 1);
            mbar_init(&a_empty[s], 1);
        }
        for (int s = 0; s < kBStages; ++s) {
            mbar_init(&b_full[s], 1);
            mbar_init(&b_empty[s], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, 256);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    const uint32_t tmem = tmem_take_q(tmem_slot, warp);
    if (GATHER) pdl_launch_dependents();          // with tensor memory in hand
    const uint32_t sbase = smem_u32(smem);
    bool ok = true;

    // No record in the list has a null blob.  The loaders and the epilogue test for it all the same: without these tests, which hold a role
    // back until its record is there, the gate/up product takes 369 us instead of 330 (6000 tokens of the 2048 x 512 layer), with
    // or without an offset in front of the list; why was not found.
    if (warp == 0) {
        // ---- MMA issuer
        if (elect_one()) {
            uint32_t kb = 0, ti = 0;
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                ok = mbar_wait(acc_empty, (ti & 1u) ^ 1u);
                if (!ok) break;
                for (int c = 0; c < n_chunk && ok; ++c, ++kb) {
                    const uint32_t sb = kb % kBStages;
                    ok = mbar_wait(&b_full[sb], (kb / kBStages) & 1u);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t bst = sbase + sb * G::kBStage, tsfb = tmem + G::kTmemSFB + sb * 32;
                    const uint64_t bd = smem_desc_sw128(bst), bs = sf_desc_q(bst + 2 * kATileQ);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
#pragma unroll
                        for (int b = 0; b < 2; ++b) sf_copy_q(tsfb + (uint32_t) (8 * k + 4 * b), bs + b * (kSFQ / 16) + k * kStepSF);
#pragma unroll
                    for (int t = 0; t < kTermsF; ++t) {
                        const uint32_t sa = (kb & 1u) * kTermsF + t;
                        ok = ok && mbar_wait(&a_full[sa], (kb >> 1) & 1u);
                        if (!ok) break;
                        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                        const uint32_t ast = sbase + G::kOffA + sa * kSlotQ, tsfa = tmem + G::kTmemSFA + sa * 16;
                        const uint64_t ad = smem_desc_sw128(ast + kSFQ), as = sf_desc_q(ast);
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            sf_copy_q(tsfa + (uint32_t) (4 * k), as + k * kStepSF);
                            mma_nvf4_q(tmem, ad + k * kStepCode, bd + k * kStepCode, G::kIdesc, tsfa + (uint32_t) (4 * k), tsfb + (uint32_t) (8 * k),
                                       (t | k) ? 1u : (c ? 1u : 0u));
                        }
                        umma_commit(&a_empty[sa]);
                    }
                    if (ok) umma_commit(&b_empty[sb]);
                }
                if (!ok) break;
                umma_commit(acc_full);
                ++ti;
            }
            if (!ok) atomicOr(a.status, 1);
        }
    } else if (warp == 1) {
        // ---- weight loader: one lane; a stage is two packed blocks (gate and up rows, or two blocks of down rows)
        if (elect_one()) {
            uint32_t kb = 0;
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                const int tile = item / n_n, n = item - tile * n_n;
                const unsigned long long bp = recs[tile].blob;
                if (bp == 0ull) continue;          // none is; see above
                const uint8_t* blob = reinterpret_cast<const uint8_t*>(bp);
                const size_t mat = (size_t) n_chunk * kBlockF;             // a 128-row block over all of K
                const uint8_t* b0 = MODE == QMODE_GU ? blob + geo.gate + n * mat : blob + geo.down + 2 * n * mat;
                const uint8_t* b1 = MODE == QMODE_GU ? blob + geo.up + n * mat : b0 + mat;
                for (int c = 0; c < n_chunk; ++c, ++kb) {
                    const uint32_t s = kb % kBStages;
                    ok = mbar_wait(&b_empty[s], ((kb / kBStages) & 1u) ^ 1u);
                    if (!ok) break;
                    const uint32_t st = sbase + s * G::kBStage, bar = smem_u32(&b_full[s]);
                    expect_bytes_q(bar, 2 * kBlockF);
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        const uint8_t* g = (b ? b1 : b0) + (size_t) c * kBlockF;
                        bulk_copy_q(st + (uint32_t) (b * kATileQ), g, kATileQ, bar);
                        bulk_copy_q(st + (uint32_t) (2 * kATileQ + b * kSFQ), g + kATileQ, kSFQ, bar);
                    }
                }
            }
            if (!ok) atomicOr(a.status, 1);
        }
    } else if (GATHER && (warp == 2 || warp == 3)) {
        // ---- activation loaders, 64 rows each.  Lane = (16-byte piece c8, row r4 of four): rows r4 + 4 i of the warp's 64; scale words:
        // lane = row, a word into each K-step's block.  Rows past the tile's last are left as they are.  A lane runs up to five slots
        // ahead of its own landed copies (of eight: the tensor core can always go on) and arrives on a slot once they are visible.
        const int64_t K = (int64_t) n_chunk * 256;
        const int lw = warp - 2, c8 = lane & 7, r4 = lane >> 3;
        uint32_t dsto[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int r7 = 4 * h + r4;
            dsto[h] = (uint32_t) (kSFQ + lw * 8 * 1024 + r7 * 128 + ((c8 ^ r7) << 4));
        }
        uint32_t issued = 0, arrived = 0;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
            const TileRec r = recs[item / n_n];
            auto image_row = [&](int row) -> size_t {
                const int i = r.row0 + min(row, r.rows - 1);
                return (size_t) (MODE == QMODE_GU ? a.src[i] : i) * kTermsF;
            };
            const uint8_t *crow[16], *srow[2];
#pragma unroll
            for (int i = 0; i < 16; ++i) crow[i] = a.img + image_row(64 * lw + 4 * i + r4) * (size_t) (K >> 1) + c8 * 16;
#pragma unroll
            for (int j = 0; j < 2; ++j) srow[j] = a.sfs + image_row(64 * lw + 32 * j + lane) * (size_t) (K >> 4);
            const int live = (r.rows - 64 * lw - r4 + 3) >> 2;         // this lane's rows are i < live
            for (int c = 0; c < n_chunk && ok; ++c)
#pragma unroll 1
                for (int t = 0; t < kTermsF; ++t) {
                    const uint32_t s = issued % kASlots;
                    ok = mbar_wait(&a_empty[s], ((issued / kASlots) & 1u) ^ 1u);
                    if (!ok) break;
                    const uint32_t slot = sbase + (uint32_t) (G::kOffA + s * kSlotQ);
                    const size_t co = (size_t) t * (size_t) (K >> 1) + (size_t) c * 128, so = (size_t) t * (size_t) (K >> 4) + (size_t) c * 16;
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (i < live) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(slot + (uint32_t) ((i >> 1) * 1024) + dsto[i & 1]), "l"(crow[i] + co) : "memory");
#pragma unroll
                    for (int j = 0; j < 2; ++j)
                        if (64 * lw + 32 * j + lane < r.rows)
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(slot + (uint32_t) (k * 512 + lane * 16 + (2 * lw + j) * 4)), "l"(srow[j] + so + 4 * k)
                                             : "memory");
                    asm volatile("cp.async.commit_group;\n" ::: "memory");
                    ++issued;
                    if (issued - arrived > 5) {
                        asm volatile("cp.async.wait_group 5;\n" ::: "memory");
                        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
                        mbar_arrive(&a_full[arrived % kASlots]);
                        ++arrived;
                    }
                }
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        for (; arrived < issued; ++arrived) mbar_arrive(&a_full[arrived % kASlots]);
        if (!ok) atomicOr(a.status, 1);
    } else if (!GATHER && warp == 2) {
        // ---- activation loader: one lane, one copy a slot
        if (elect_one()) {
            uint32_t ka = 0;
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                const TileRec r = recs[item / n_n];
                if (r.blob == 0ull) continue;
                const uint32_t bytes = (uint32_t) tile_units(r.rows) * 1024u;
                const uint8_t* g = a.img + image_block(r, n_chunk, 0, 0);
                for (int i = 0; i < n_chunk * kTermsF; ++i, ++ka, g += bytes) {
                    const uint32_t s = ka % kASlots;
                    ok = mbar_wait(&a_empty[s], ((ka / kASlots) & 1u) ^ 1u);
                    if (!ok) break;
                    const uint32_t bar = smem_u32(&a_full[s]);
                    expect_bytes_q(bar, bytes);
                    bulk_copy_q(sbase + (uint32_t) (G::kOffA + s * kSlotQ), g, bytes, bar);
                }
            }
            if (!ok) atomicOr(a.status, 1);
        }
    } else if (warp >= 4) {
        // ---- epilogue: thread p reads TMEM lane p (= tile row p), warps 4-7 the first and 8-11 the second half of the item's
        // columns.  A warp may only read lanes 32 (warp % 4) .. + 31.  All of a thread's 128 values go to registers first, so the
        // one accumulator is back with the tensor core before any of them is worked on.
        const int p = (warp & 3) * 32 + lane, half = warp >= 8 ? 1 : 0;
        const uint32_t tbase = tmem + ((uint32_t) ((warp & 3) * 32) << 16);
        const bool wide = MODE == QMODE_GU || (reinterpret_cast<uintptr_t>(a.dm) & 31) == 0;
        uint32_t ti = 0;
        for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
            const int tile = item / n_n, n = item - tile * n_n;
            const TileRec r = recs[tile];
            if (r.blob == 0ull) continue;
            const bool row_live = p < r.rows;
            const float* tail = reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(r.blob) + geo.tail);
            const int64_t ir = !row_live ? 0 : (MODE == QMODE_GU ? (int64_t) a.src[r.row0 + p] : (int64_t) (r.row0 + p));
            const float f = row_live ? a.inv[ir] : 0.f;
            const float sg = tail[0] * f, su = tail[1] * f, sd = tail[2] * f;
            ok = __all_sync(kFull, mbar_wait(acc_full, ti & 1u));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            uint32_t v[4][32];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int col = MODE == QMODE_GU ? (i >> 1) * 128 + half * 64 + (i & 1) * 32 : half * 128 + i * 32;
                tmem_ld32(tbase + (uint32_t) col, v[i]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            mbar_arrive(acc_empty);
            ++ti;
            if (!row_live) continue;
            if (MODE == QMODE_GU) {
                float* hrow = a.h + (size_t) (r.row0 + p) * a.L.n_ff + n * 128 + half * 64;
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float o[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) o[e] = swiglu(__uint_as_float(v[i][8 * j + e]) * sg, __uint_as_float(v[2 + i][8 * j + e]) * su, a.L);
                        store8_q(hrow + 32 * i + 8 * j, o, wide);
                    }
            } else {
                float* orow = a.dm + (size_t) (r.row0 + p) * a.L.n_embd + n * 256 + half * 128;
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        float o[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) o[e] = __uint_as_float(v[i][8 * j + e]) * sd;
                        store8_q(orow + 32 * i + 8 * j, o, wide);
                    }
            }
        }
        if (!ok && lane == 0) atomicOr(a.status, 1);
    }
    tmem_give_q(tmem, warp);
}

// ---------------------------------------------------------------- down product with the tile's rows resident
// When n_ff <= 512 a tile's SwiGLU rows - 128 rows x n_ff columns as four FP4 terms, 72 KB per 256 columns with their scale
// words - fit in shared memory for the whole tile, so they are fetched once instead of once per block of down rows, and the
// kernel streams only weights: one bulk copy a stage brings a block of 128 down rows over all of K (KC packed blocks, which
// are consecutive in the blob).  Item = a 128-row tile; per tile 16 x (n_embd / 2048) stages, each one accumulator of 128
// columns, two accumulators in flight.  Tensor memory: accumulators [0, 256), the tile's activation scales [256, 256 + 64 KC),
// per stage the weight scales.
template <int KC>
struct GeoR {
    static constexpr int kOffB = KC * kTermsF * kSlotQ;             // [chunk][term] slots, then two stages of KC packed blocks
    static constexpr int kStageB = KC * kBlockF;
    static constexpr int kBars = kOffB + 2 * kStageB;
    static constexpr size_t kSmem = 1024 + (size_t) kBars + 256;
    static constexpr uint32_t kTmemSFA = 256, kTmemSFB = 256 + 64 * KC, kSFBStage = 16 * KC;
    static constexpr uint32_t kIdesc = (1u << 7) | (1u << 10) | ((uint32_t) (128 >> 3) << 17) | ((uint32_t) (128 >> 4) << 24);
};

template <int KC>
__global__ void __launch_bounds__(kThreadsQ, 1) prefill_down_resident_kernel(PrefillFArgs a) {
    using G = GeoR<KC>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t) 1023);
    uint64_t* b_full = reinterpret_cast<uint64_t*>(smem + G::kBars);
    uint64_t* b_empty = b_full + 2;
    uint64_t* acc_full = b_empty + 2;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* a_full = acc_empty + 2;
    uint64_t* a_empty = a_full + 1;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(a_empty + 1);

    const int warp = warp_index(), lane = threadIdx.x & 31;
    const int n_nb = (int) (a.L.n_embd / 128);            // blocks of 128 down rows = stages per tile
    const TileRec* recs = a.recs + first_tile(a.from);
    const int n_tiles = *a.to - first_tile(a.from);
    const PackedGeom geo = packed_geom(a.L.n_embd, a.L.n_ff);

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&b_full[s], 1);
            mbar_init(&b_empty[s], 1);
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], 256);
        }
        mbar_init(a_full, 1);
        mbar_init(a_empty, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    const uint32_t tmem = tmem_take_q(tmem_slot, warp);
    const uint32_t sbase = smem_u32(smem);
    bool ok = true;

    if (warp == 0) {
        if (elect_one()) {
            uint32_t ti = 0, nbc = 0;
            for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
                ok = mbar_wait(a_full, ti & 1u);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                // the tile's activation scales: shared -> tensor memory, once
#pragma unroll
                for (int q = 0; q < KC * kTermsF; ++q) {
                    const uint64_t as = sf_desc_q(sbase + (uint32_t) (q * kSlotQ));
#pragma unroll
                    for (int k = 0; k < 4; ++k) sf_copy_q(tmem + G::kTmemSFA + (uint32_t) (16 * q + 4 * k), as + k * kStepSF);
                }
                const uint64_t ad = smem_desc_sw128(sbase + kSFQ);
                for (int nb = 0; nb < n_nb; ++nb, ++nbc) {
                    const uint32_t s = nbc & 1u, par = (nbc >> 1) & 1u;
                    ok = mbar_wait(&acc_empty[s], par ^ 1u);
                    if (ok) ok = mbar_wait(&b_full[s], par);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t sb = sbase + (uint32_t) G::kOffB + s * G::kStageB;
                    const uint32_t tsfb = tmem + G::kTmemSFB + s * G::kSFBStage;
                    const uint32_t d = tmem + s * 128;
#pragma unroll
                    for (int c = 0; c < KC; ++c) {
                        const uint64_t bd = smem_desc_sw128(sb + (uint32_t) (c * kBlockF)), bs = sf_desc_q(sb + (uint32_t) (c * kBlockF + kATileQ));
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            sf_copy_q(tsfb + (uint32_t) (16 * c + 4 * k), bs + k * kStepSF);
#pragma unroll
                            for (int t = 0; t < kTermsF; ++t)
                                mma_nvf4_q(d, ad + (uint64_t) ((c * kTermsF + t) * (kSlotQ / 16)) + k * kStepCode, bd + k * kStepCode, G::kIdesc,
                                           tmem + G::kTmemSFA + (uint32_t) (64 * c + 16 * t + 4 * k), tsfb + (uint32_t) (16 * c + 4 * k), (c | k | t) ? 1u : 0u);
                        }
                    }
                    umma_commit(&b_empty[s]);
                    umma_commit(&acc_full[s]);
                }
                if (!ok) break;
                umma_commit(a_empty);       // the resident rows may be replaced once every MMA of the tile has read them
                ++ti;
            }
            if (!ok) atomicOr(a.status, 1);
        }
    } else if (warp == 1) {
        if (elect_one()) {
            uint32_t nbc = 0;
            for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
                const uint8_t* down = reinterpret_cast<const uint8_t*>(recs[tile].blob) + geo.down;
                for (int nb = 0; nb < n_nb; ++nb, ++nbc) {
                    const uint32_t s = nbc & 1u;
                    ok = mbar_wait(&b_empty[s], ((nbc >> 1) & 1u) ^ 1u);
                    if (!ok) break;
                    const uint32_t bar = smem_u32(&b_full[s]);
                    expect_bytes_q(bar, (uint32_t) G::kStageB);
                    bulk_copy_q(sbase + (uint32_t) G::kOffB + s * G::kStageB, down + (size_t) nb * G::kStageB, (uint32_t) G::kStageB, bar);
                }
            }
            if (!ok) atomicOr(a.status, 1);
        }
    } else if (warp == 2) {
        // ---- the tile's rows: one copy per (chunk, term)
        if (elect_one()) {
            uint32_t ti = 0;
            for (int tile = blockIdx.x; tile < n_tiles && ok; tile += gridDim.x) {
                const TileRec r = recs[tile];
                ok = mbar_wait(a_empty, (ti & 1u) ^ 1u);
                if (!ok) break;
                const uint32_t bytes = (uint32_t) tile_units(r.rows) * 1024u, bar = smem_u32(a_full);
                expect_bytes_q(bar, (uint32_t) (KC * kTermsF) * bytes);
                const uint8_t* g = a.img + image_block(r, KC, 0, 0);
#pragma unroll
                for (int q = 0; q < KC * kTermsF; ++q) bulk_copy_q(sbase + (uint32_t) (q * kSlotQ), g + (size_t) q * bytes, bytes, bar);
                ++ti;
            }
            if (!ok) atomicOr(a.status, 1);
        }
    } else if (warp >= 4) {
        // ---- epilogue: thread p = tile row p reads TMEM lane p of each finished accumulator, half of its 128 columns
        const int p = (warp & 3) * 32 + lane, half = warp >= 8 ? 1 : 0;
        const uint32_t tbase = tmem + ((uint32_t) ((warp & 3) * 32) << 16) + (uint32_t) (half * 64);
        const bool wide = (reinterpret_cast<uintptr_t>(a.dm) & 31) == 0;
        uint32_t nbc = 0;
        for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
            const TileRec r = recs[tile];
            const bool row_live = p < r.rows;
            const float* tail = reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(r.blob) + geo.tail);
            const float sd = row_live ? tail[2] * a.inv[r.row0 + p] : 0.f;
            const int w0 = (warp & 3) * 32;
            float* orow = a.dm + (size_t) (r.row0 + w0) * a.L.n_embd + half * 64;
            for (int nb = 0; nb < n_nb; ++nb, ++nbc) {
                const uint32_t s = nbc & 1u;
                ok = __all_sync(kFull, mbar_wait(&acc_full[s], (nbc >> 1) & 1u));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                uint32_t v[2][32];
                tmem_ld32(tbase + s * 128, v[0]);
                tmem_ld32(tbase + s * 128 + 32, v[1]);
                asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
                mbar_arrive(&acc_empty[s]);
                if (w0 >= r.rows) continue;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    float o[32];
#pragma unroll
                    for (int e = 0; e < 32; ++e) o[e] = __uint_as_float(v[i][e]) * sd;
                    store_rows32_q(orow + nb * 128 + 32 * i, (size_t) a.L.n_embd, r.rows - w0, lane, o, wide);
                }
            }
            if (!ok) break;
        }
        if (!ok && lane == 0) atomicOr(a.status, 1);
    }
    tmem_give_q(tmem, warp);
}

template <int KC>
int32_t launch_down_resident(const PrefillFArgs& a, cudaStream_t st) {
    static std::atomic<bool> configured[64];   // per device; threads of different devices call concurrently
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return (int32_t) cudaErrorInvalidDevice;
    if (!configured[dev].load(std::memory_order_acquire)) {
        const cudaError_t e = cudaFuncSetAttribute(prefill_down_resident_kernel<KC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) GeoR<KC>::kSmem);
        if (e != cudaSuccess) return (int32_t) e;
        configured[dev].store(true, std::memory_order_release);
    }
    prefill_down_resident_kernel<KC><<<(unsigned) sm_count(), kThreadsQ, GeoR<KC>::kSmem, st>>>(a);
    return launch_status();
}

size_t al256q(size_t v) { return (v + 255) & ~(size_t) 255; }

template <int MODE, bool GATHER>
int32_t launch_q(const PrefillFArgs& a, cudaStream_t st) {
    static std::atomic<bool> configured[64];   // per device; threads of different devices call concurrently
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return (int32_t) cudaErrorInvalidDevice;
    if (!configured[dev].load(std::memory_order_acquire)) {
        const cudaError_t e = cudaFuncSetAttribute(prefill_nvf4_kernel<MODE, GATHER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) GeoQ::kSmem);
        if (e != cudaSuccess) return (int32_t) e;
        configured[dev].store(true, std::memory_order_release);
    }
    if (GATHER) launch_k(prefill_nvf4_kernel<MODE, GATHER>, dim3((unsigned) sm_count()), dim3(kThreadsQ), GeoQ::kSmem, st, a);
    else prefill_nvf4_kernel<MODE, GATHER><<<(unsigned) sm_count(), kThreadsQ, GeoQ::kSmem, st>>>(a);
    return launch_status();
}

}  // namespace
}  // namespace bsx

using namespace bsx;

// Rows an expert, on average over the call, up to which the decode stream takes it.  Whole layer, bf16 rows, back to back, stream against tiles: 2048 x 512 with
// 512 + 1 experts at 1.4 rows an expert 207 : 310 us, 16.7 338 : 498, 32 443 : 547, 47 567 : 604; 5120 x 2304 with 384 + 1 at 14
// rows 1500 : 2411, 27 2103 : 2780; 7168 x 2048 with 256 + 1 at 17.5 rows 1473 : 2203, 35 2112 : 2437.
constexpr int64_t kShortRows = 48;

// Rows of up to 1025 experts make at most this many tiles.
static int64_t prefill_cap_tiles(int64_t cap_rows, int64_t n_expert) { return std::min(cap_rows, cap_rows / 128 + std::min<int64_t>(n_expert, 1025)); }

// Where a call's buffers lie in its scratch, and the route that its numbers choose.
struct PrefillCarve {
    bool stream;                       // few rows an expert: the decode stream
    int64_t cap_recs, cap_items, slab_units;
    int n_slabs;
    size_t xcodes, xsf, xinv, h, img, hcodes, hsf, hinv, recs, slabs, items, n_items, bytes;
};
// n_held of the n_expert experts have blobs here.  Where that is not all of them, the tile images have room for twice an even share
// of the rows, and what a skewed routing sends beyond it is done in further slabs over the same room (kernels of a slab without
// tiles return at once).
static PrefillCarve prefill_carve(const bsx_expert_layout& L, int64_t n_tokens, int64_t cap_rows, int64_t n_expert, int64_t n_held) {
    PrefillCarve c = {};
    const int64_t H = L.n_embd, I = L.n_ff;
    c.stream = cap_rows <= kShortRows * n_expert && n_tokens <= 0x7FFFFFFF;
    c.cap_recs = prefill_cap_tiles(cap_rows, n_held);
    c.cap_items = cap_rows / kPassEntries + c.cap_recs;
    const int64_t all = image_units(cap_rows, c.cap_recs);
    const int64_t share = n_held < n_expert ? std::min(cap_rows, (2 * cap_rows * n_held + n_expert - 1) / n_expert) : cap_rows;
    c.slab_units = std::max<int64_t>(kMaxUnits, std::min(all, image_units(share, prefill_cap_tiles(share, n_held))));
    c.n_slabs = c.stream ? 1 : (int) ((all + c.slab_units - 1) / c.slab_units);
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
    if (c.stream) {
        c.hcodes = take((size_t) cap_rows * kTermsF * I / 2);
        c.hsf = take((size_t) cap_rows * kTermsF * I / 16);
        c.items = take((size_t) c.cap_items * sizeof(PassRec));
        c.n_items = take(4);
    } else {
        at = (at + 4095) & ~(size_t) 4095;
        c.img = take((size_t) (c.slab_units + kMaxUnits) * 1024 * kTermsF * ((H + I) / 256));
    }
    c.hinv = take((size_t) (cap_rows + 128) * 4);
    c.recs = take((size_t) c.cap_recs * sizeof(TileRec));
    c.slabs = take((size_t) (c.n_slabs + 1) * 4);
    c.bytes = at;
    return c;
}

extern "C" size_t bsx_experts_prefill_packed_held_scratch_bytes(const bsx_expert_layout* L, int64_t n_tokens, int64_t cap_rows, int32_t n_expert, int32_t n_held) {
    if (!L || n_tokens < 0 || cap_rows < 0 || n_expert < 1 || n_held < 0 || n_held > n_expert || !bsx_expert_packed_bytes(L)) return 0;
    return prefill_carve(*L, n_tokens, cap_rows, n_expert, n_held).bytes;
}

// the most that any number of experts needs: the stream's for all of them, the tiles' for the largest number that goes to tiles
extern "C" size_t bsx_experts_prefill_packed_scratch_bytes(const bsx_expert_layout* L, int64_t n_tokens, int64_t cap_rows) {
    if (!L || n_tokens < 0 || cap_rows < 0 || !bsx_expert_packed_bytes(L)) return 0;
    const int64_t many = std::max<int64_t>(1025, (cap_rows + kShortRows - 1) / kShortRows);
    const int64_t tiled = n_tokens > 0x7FFFFFFF ? 1025 : std::min<int64_t>(1025, (cap_rows - 1) / kShortRows);
    const size_t a = prefill_carve(*L, n_tokens, cap_rows, many, many).bytes;
    return tiled < 1 ? a : std::max(a, prefill_carve(*L, n_tokens, cap_rows, tiled, tiled).bytes);
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
    uint8_t *xcodes = base + c.xcodes, *xsf = base + c.xsf;
    float *xinv = reinterpret_cast<float*>(base + c.xinv), *h = reinterpret_cast<float*>(base + c.h), *hinv = reinterpret_cast<float*>(base + c.hinv);
    RecordArgs ra;
    ra.tiles = tiles;
    ra.n_tiles = n_tiles;
    ra.off = off;
    ra.blob_table = blob_table;
    ra.cap_tiles = cap_tiles;
    ra.recs = reinterpret_cast<TileRec*>(base + c.recs);
    ra.cap_recs = c.cap_recs;
    ra.slab_first = reinterpret_cast<int32_t*>(base + c.slabs);
    ra.n_slabs = c.n_slabs;
    ra.slab_units = c.slab_units;
    ra.items = nullptr;
    ra.n_items = nullptr;
    ra.cap_items = c.cap_items;
    ra.pass_entries = cap_rows > kPassEntries / 2 * n_expert ? 2 * kPassEntries : kPassEntries;
    ra.tile_items = (int) (I / 128);
    ra.sm_count = sm_count();
    ra.status = status;
    PrefillFArgs a;
    a.L = L;
    a.recs = ra.recs;
    a.from = nullptr;
    a.to = ra.slab_first + 1;
    a.src = src;
    a.sfs = nullptr;
    a.h = h;
    a.dm = dm;
    a.status = status;
    // Few rows an expert: a tile's 128 tensor-core rows would be mostly padding and cost twice what the weights' bytes do, so the rows
    // go through the decode stream instead (experts_nvf4.cu: passes of 8 or 16 rows as the MMA's narrow side, bound by the weights),
    // crowded tiles aside (tile_records_kernel), which in most calls there are none of: their kernels then return at once.
    if (c.stream) {
        PdlScope pdl(true, 1);      // the first kernel follows the caller's work
        ra.items = reinterpret_cast<PassRec*>(base + c.items);
        ra.n_items = reinterpret_cast<int*>(base + c.n_items);
        launch_k(tile_records_kernel, dim3(1), dim3(1024), 0, st, ra);
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
        packed_x_images(x, x_kind, n_tokens, H, xcodes, xsf, xinv, st);
        a.img = xcodes;
        a.sfs = xsf;
        a.inv = xinv;
        int32_t rc = launch_q<QMODE_GU, true>(a, st);
        if (rc == BSX_OK) rc = packed_pass_product(false, e, ra.items, ra.n_items, ra.pass_entries, xcodes, xsf, xinv, status, st);
        if (rc != BSX_OK) return rc;
        uint8_t *hcodes = base + c.hcodes, *hsf = base + c.hsf;
        packed_listed_images(h, ra.items, ra.n_items, ra.pass_entries, ra.recs, ra.slab_first, I, hcodes, hsf, hinv, st);
        a.img = hcodes;
        a.sfs = hsf;
        a.inv = hinv;
        rc = launch_q<QMODE_DOWN, true>(a, st);
        if (rc != BSX_OK) return rc;
        return packed_pass_product(true, e, ra.items, ra.n_items, ra.pass_entries, hcodes, hsf, hinv, status, st);
    }
    uint8_t *ximg = base + c.img, *himg = ximg + (size_t) (c.slab_units + kMaxUnits) * 1024 * kTermsF * (H / 256);
    const TileRec* recs = ra.recs;
    const int32_t* slabs = ra.slab_first;
    tile_records_kernel<<<1, 1024, 0, st>>>(ra);
    if (H <= 2048) prefill_images_kernel<128><<<(unsigned) ((n_tokens + 1) / 2), 256, 0, st>>>(x, x_kind, n_tokens, H, xcodes, xsf, xinv);
    else prefill_images_kernel<256><<<(unsigned) n_tokens, 256, 0, st>>>(x, x_kind, n_tokens, H, xcodes, xsf, xinv);
    // a tile takes three units at least, and one may begin in a slab's last unit
    const int64_t slab_tiles = std::min(std::min(cap_tiles, c.cap_recs), c.slab_units / 3 + 1);
    for (int s = 0; s < c.n_slabs; ++s) {
        a.from = s ? slabs + s : nullptr;
        a.to = slabs + s + 1;
        for (int64_t t0 = 0; t0 < slab_tiles; t0 += 65535)
            tile_images_kernel<<<dim3((unsigned) (H / 256), (unsigned) std::min<int64_t>(slab_tiles - t0, 65535)), 256, 0, st>>>(recs, a.from, a.to, (int) t0, src, xcodes, xsf, H,
                                                                                                                                 ximg);
        a.img = ximg;
        a.inv = xinv;
        int32_t rc = launch_q<QMODE_GU, false>(a, st);
        if (rc != BSX_OK) return rc;
        const unsigned hb = (unsigned) (slab_tiles * 16);
        a.img = himg;
        if (I <= 512) h_images_kernel<1><<<hb, 256, 0, st>>>(recs, a.from, a.to, h, I, himg, hinv);
        else h_images_kernel<0><<<hb, 256, 0, st>>>(recs, a.from, a.to, h, I, himg, hinv);
        a.inv = hinv;
        // n_ff <= 512: the tile's rows stay in shared memory and only weights stream
        rc = I == 256 ? launch_down_resident<1>(a, st) : I == 512 ? launch_down_resident<2>(a, st) : launch_q<QMODE_DOWN, false>(a, st);
        if (rc != BSX_OK) return rc;
    }
    return BSX_OK;
}

extern "C" int32_t bsx_experts_prefill_packed(const bsx_expert_layout* layout, const unsigned long long* blob_table, const int32_t* off,
                                              const int32_t* src, const int32_t* tiles, const int32_t* n_tiles, int64_t cap_tiles, int64_t cap_rows,
                                              const void* x, int32_t x_kind, int64_t n_tokens, int32_t n_expert, void* scratch, float* dm, int32_t* status,
                                              void* stream) {
    return bsx_experts_prefill_packed_held(layout, blob_table, off, src, tiles, n_tiles, cap_tiles, cap_rows, x, x_kind, n_tokens, n_expert, n_expert, scratch, dm,
                                           status, stream);
}
