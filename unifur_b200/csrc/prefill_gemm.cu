// Prefill path: y[M, N] = x * dequant(W)^T (+bias) (+ s * (x A^T) B^T) for many rows of x,
// W stored as packed NF4 [N, K] with 64-blocks along K.  A dense contraction: tensor-core
// bound, built on tcgen05.mma with the dequantised weight operand and the accumulator in
// tensor memory (TMEM) and the activations in shared memory.
//
// Two CTAs of a cluster, one per SM, work on a tile of 256 weight rows x 256 activation rows together
// (cta_group::2): each holds 128 weight rows and their accumulators in its tensor memory and half of the
// activations in its shared memory, which halves what a shared memory is written and read per
// multiplication.  Few rows take tiles of 128 activation rows (share_tiles).  K goes in steps of two stages of 64; what warps
// hand to one another they hand over a step at a time.  Roles inside a CTA (persistent, 864 threads):
//   warp 0      TMA producer: this CTA's half of a step's x tiles [128 rows x 64 k] (f16, 128B-swizzled,
//               K-major) into a 96 KB ring of steps; after the K loop the same ring carries the LoRA
//               intermediate T (bf16 hi / lo halves) and, a slot before it, the matching
//               128 x 64 tile of LoRA B, so the adapter is just more steps (with both
//               operands in shared memory).
//   warp 1      owns TMEM (alloc/dealloc); in the even CTA it issues the pair's tcgen05.mma.
//   warp 6      asks for the packed codes, 128 weight rows x 128 a step by TMA, prefetched into L2, and for their scales.
//   warps 2-5, 23-26  epilogue: TMEM -> registers -> (* row scale, + bias) -> bf16/f32 ->
//               shared -> TMA store.
//   warps 7-22  dequantisers, four groups of 128 threads, two to a step in turn.  A thread
//               owns one weight row (= one TMEM lane; a warp may only touch the lane quarter its
//               number names): it takes the row's 32 packed bytes of a stage from shared memory, looks byte by
//               byte a pair of levels up in a table, multiplies by the block's scale in f16x2 and writes the
//               64 f16 values into its lane of a ring of four steps of TMEM columns with tcgen05.st.
//
// Why the weight operand lives in TMEM.  The table look-ups, the TMA and the MMA's reads of the
// activations already take most of the 128 B/clk a shared memory delivers; the dequantised weight never
// touches it.  The price: the accumulator
// (256 columns) and the weight ring (8 x 32 columns) share the 512 TMEM columns, so there is one
// accumulator and the MMAs of the next tile wait while the epilogue reads it out.
//
// What bounds it: a wide tile's MMAs, 1024 cycles a step of 256 columns (893 measured for the 896 of 224), and for many rows
// the clock that the power limit leaves (1.4 GHz on random operands).  A narrow tile's step is the dequantisers' latency, 0.4 us.
// With a stage at a time the skeleton alone, no look-ups, no stores, a quarter of the MMAs, took 0.29 us a stage: the one lane that
// asked for the activations spent 300 to 440 cycles on each, and scales loaded by the threads another 0.05 us.  Before ->
// now, whole calls, weights and inputs in turn: 64 x 4096 x 4096 20.5 -> 18.0 us, 128 x 8192 x 8192 38.3 -> 31.3, 203 x 3584 x 18944 35.7 ->
// 34.3, 512 x 4096 x 4096 31.6 -> 26.8, 64 x 14336 x 4096 36.0 -> 31.0; 256 x 4096 x 4096 25.0 -> 25.5; 2048 x 4096 x 14336 within what runs
// differ (205 to 210); the GEMM of a backward over 2048 x 4096 x 14336 167 -> 147.  What got slower: few stages a tile in several rounds of
// tiles with u8 scales loaded by the threads, 3216 x 512 x 4160 34.1 -> 35.1, 531 x 512 x 19200 36.1 -> 37.2.
// The start counts for few rows: most CTAs start when the pre-pass's end, so the codes of the first steps are asked for
// before anything else is set up: 512 x 4096 x 4096 19.4 -> 17.6 us of the kernel.  The CTAs of a pair meet with a release and an acquire by
// all threads, at the start and at the end (relaxed arrivals took 0.5 to 0.9 us a call less).
//
// The MMA computes D[n, m] = sum_k W[n, k] x[m, k]: weight rows are the MMA's M (TMEM lanes),
// activation rows its N (256 accumulator columns).  Both operands are f16 with f32 accumulation:
// rounding the dequantised weight to bf16 instead would cost ~1.6e-3 relative error, above the
// 1e-3 parity bar, while f16 costs ~3e-4.  The bf16 activations are converted to f16 by a
// pre-pass, divided by a power of two that the epilogue multiplies back: exact where f16 holds the value's
// eight bits, which is down to 2^-31 of the row's largest magnitude where the row has its own power of two,
// and down to 2^-17 where it has none (the pre-pass says which rows that is).  It also
// produces the LoRA intermediate.
//
// The other orientation (W [K][N] with the 64-blocks along N, the reference's own; f32 or bf16
// activations) comes through the same GEMM at more than 16 rows: small kernels beside the pre-pass write the
// transposed nibbles, the scales as f16 [N / 64][K] and the adapter factors in this kernel's
// orientation into the workspace (the nibbles exactly; the scales with the rounding the dequantisers
// apply anyway).  A weight row's scale then changes with every k, and is the same for 64 rows: a step's scales come by TMA
// beside its codes, and every lane reads the same pairs (kScalesPerK).  f32 activations are converted to f16
// directly, every row divided by its own power of two.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <mutex>
#include <type_traits>

#include "kernels.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace nf4 {

__device__ int g_prefill_error = 0;  // set when a bounded wait gives up
__device__ int *g_prefill_error_host = nullptr;  // the same, in mapped host memory (set by the host-pointer entry points)

namespace {

constexpr int BM = 128;        // weight rows per CTA and tile (half of the pair's MMA M; TMEM lanes)
constexpr int BK = 64;         // k per stage = one quantization block = one 128B swizzle row
constexpr int kASteps = 4;     // TMEM ring of dequantised weights: steps of two stages
constexpr int kStageCols = BK / 2;  // 32 columns: two f16 per 32-bit cell
constexpr int kAccCols = 256;  // the accumulator: columns [0, 256); the weight ring follows
constexpr int kTmemCols = 512;
constexpr int kBarRing = 8;    // steps whose barriers are told apart (more than the deepest ring of activations holds)
constexpr int kCodeSlots = 3;  // shared-memory ring of packed weight codes, a step each
constexpr int kCodeTileBytes = BM * 64;        // 8 KB: 128 weight rows x 128 codes, written by TMA (64B swizzle)
constexpr int kScaleTileBytes = BM * 16;       // 2 KB: the same rows' scales of four stages (f32) or sixteen (u8), by TMA
constexpr int kPerKBytes = BM / 64 * 2 * BK * 2;  // 512 bytes: a scale for every k of a step and 64-block of rows
constexpr int kLoraTileBytes = BM * BK * 2;    // 16 KB: 128 rows of LoRA B x 64 ranks, written by TMA

constexpr int kEpiBytes = 32 * 1024;       // output staging: half a wide tile of bf16 (as two swizzled boxes), a quarter of f32
constexpr int kThreads = 27 * 32;
constexpr int kFirstExpanderWarp = 7;      // sixteen warps
constexpr int kFirstEpilogueWarpB = 23;    // the second set of four epilogue warps
constexpr int kCodeWarp = 6;               // asks for the packed codes
constexpr int kStepWarps = 16;             // warps that dequantise a step: two groups in each CTA
constexpr int kExpanderGroups = 4;         // of four warps (one per TMEM lane quarter) each
constexpr uint64_t kInOutMinRows = 17;     // the other weight orientation comes here from this many rows on

// Places in the shared window.  The lookup table starts at 0x10000, so that one byte permute of the code
// word with {4 lane, 0, 1, rank} is an entry's address; the first third of the ring of activations lies below it.
constexpr uint32_t kBarsAt = 0x800, kTmemSlotAt = 0xa00, kRowScalesAt = 0xc00, kCodesAt = 0x1000, kXAt = 0x8000, kTableAt = 0x10000,
                   kEpiAt = 0x20000, kXRestAt = 0x28000, kScalesRestAt = kXRestAt + 2 * (kTableAt - kXAt), kScalesAt = kCodesAt + kCodeSlots * kCodeTileBytes,
                   kWindowEnd = kScalesRestAt + kScaleTileBytes;
constexpr uint32_t kDynamicSmem = kWindowEnd - 1024;   // the dynamic shared memory starts at 1024 or a little above
static_assert(kScalesAt + (kCodeSlots - 1) * kScaleTileBytes <= kXAt && kEpiAt + kEpiBytes <= kXRestAt, "places overlap");
static_assert(kDynamicSmem <= 227 * 1024, "shared memory");

// The ring of activations, in slots of a step: this CTA's half of two stages' tiles of BN rows.  96 KB of 32 or 16 KB each.
template <int BN>
struct XRing {
    static constexpr uint32_t kTile = BN / 2 * BK * 2, kSlot = 2 * kTile, kBelow = (kTableAt - kXAt) / kSlot, kSlots = 3 * kBelow;
    static_assert(kSlot >= kLoraTileBytes && kSlots < kBarRing, "the adapter's tile takes a slot; a parity names a step's round");
    __device__ static __forceinline__ uint32_t place(uint32_t slot) {
        return kXAt + slot * kSlot + (slot >= kBelow ? kXRestAt - kTableAt : 0u);
    }
    __device__ static __forceinline__ uint32_t next(uint32_t slot) { return slot + 1 == kSlots ? 0u : slot + 1; }
};

// How the dequantisers get a row's scale of a stage: loaded by the thread, three of its stages ahead; by TMA, sixteen bytes of every row
// with the codes of a step; or, for weights in the other orientation, a scale for every k, a step's 128 pairs of each of the CTA's two
// 64-blocks of rows (handed round with shuffles, 32 a stage beside as many lookups, a narrow tile's stage took 0.31 us).  A warp's
// loads of 32 rows' scales are 32 sectors for four bytes of each, and its walk to the next one some forty instructions: 64 x 16384 x
// 18944 67 us with them, 55 without scales.  TMA takes rows of whole 16-byte pieces only: d_in a multiple of 256 (u8: 1024).
enum ScaleSource : int { kScalesLoaded = 0, kScalesTma = 1, kScalesPerK = 2 };
__device__ __forceinline__ uint32_t scales_place(uint32_t slot) {
    return slot + 1 == kCodeSlots ? kScalesRestAt : kScalesAt + slot * kScaleTileBytes;
}

// barrier slots
// Full counts, in the even CTA, what a step of the pair needs: both halves of the activations (or of an
// adapter step's operands) and the sixteen warps of both CTAs that dequantise its weights.  Done is a step's
// MMAs over, in both CTAs: whatever the step's slots held is free.  Steps number on over a pair's segments,
// the adapter's included; step c has barriers c % kBarRing and weight columns c % kASteps.
constexpr int kBarFull = 0, kBarDone = kBarFull + kBarRing, kBarAccFull = kBarDone + kBarRing, kBarAccEmpty = kBarAccFull + 1,
              kBarCFull = kBarAccEmpty + 1, kBarCEmpty = kBarCFull + 2 * kCodeSlots, kNumBars = kBarCEmpty + kCodeSlots;
static_assert(kBarsAt + kNumBars * 8 <= kTmemSlotAt, "barrier room");

// Where the codes of a main step go.  Blocks number on over a pair's segments, without the adapter's steps.  A slot's rounds are told
// apart by two barriers in turn: a warp that dequantises takes every other step, so that it does not see every round of a slot, and
// with one barrier a slot a wait for block b passed at once, with the parity of b - 6, while b - 3 was still under way.  The barrier of
// block b had block b - 6 before; that one has landed whenever a warp comes to wait for b: at its turn before this one, two steps
// back, it waited for the MMAs of the step four before that.
struct CodePlace {
    uint32_t slot, full, parity;  // of the ring, its barrier among the kBarCFull ones, the parity of the block's round on it
};
__host__ __device__ __forceinline__ CodePlace code_place(uint32_t block) {
    const uint32_t round = block / kCodeSlots, slot = block - round * kCodeSlots;
    return {slot, slot + (round & 1u) * kCodeSlots, (round >> 1) & 1u};
}

struct PrefillParams {
    const uint8_t *codes;
    const float *absmax;
    const uint8_t *scale_codes;
    const float *scale_of_scales;
    const float *bias;
    const float *row_scale;       // [M] power-of-two factor each activation row was divided by
    // Weights that came in the other orientation ([d_in][d_out], blocks along d_out) are repacked
    // before the GEMM: `codes` then holds the transposed nibbles, and a weight's scale depends on
    // k, not on the k-stage: scales_t[n / 64][k] as f16, already divided by the weight's power of two.
    const __half *scales_t;
    uint32_t M, N, K, rank;
    uint32_t lora_chunks;  // ceil(rank / 64); T is [M][2 * 64 * lora_chunks] (hi halves, then lo)
    uint32_t m_tiles;
    uint32_t box_rows;     // activation rows a CTA brings of a tile
    // Work of a pair of CTAs (tiles of 256 weight rows x BN activation rows, the even CTA the lower 128
    // weight rows): first its share of the `sk_tiles` tiles whose k-stages all pairs divide
    // evenly between them (a tile can be split between neighbouring pairs), then `dp_rounds`
    // whole tiles.  A pair that multiplies the leading stages of a tile leaves its accumulators
    // in `partial` ([CTA][BN][BM] f32) and raises its CTAs' words of `sk_flags`; the pair that multiplies
    // the last stages adds those and finishes the tile.
    // split > 1 (fewer tiles than pairs): a tile is `split` pairs' instead, an equal part of its stages each; all leave
    // their accumulators in `partial`, and a kernel of its own adds them (sum_parts_kernel).
    uint32_t sk_tiles, dp_rounds, split;
    uint32_t share_r;      // main stages of the shared tiles beyond share_q for every pair (a division in 64 bits takes the
    uint64_t share_q;      // kernel's start 0.2 us)
    float *partial;
    uint32_t *sk_flags;
    uint32_t wait_ns;  // bound of the wait for a neighbour's flag
    // A TMA store writes whole 16-byte pieces: the piece that holds the last columns would reach beyond them into the
    // row's padding, which is not the call's.  Where d_out ends inside a piece, the tiles at that end are stored plainly.
    void *y_ragged;    // the output then, else null
    uint64_t ldy;
};

// A pair's list of segments (tile, main k-stages [b, e)), in the order they are worked on: the
// shared tiles from the last to the first -- a piece without a tile's last stage comes first and
// waits for nobody; the piece with the last stage of a tile that a neighbour began comes last of
// them -- then the whole tiles.
struct WorkList {
    uint64_t u0, u1;   // this pair's range of main stages of the shared tiles
    uint32_t ks;       // main stages per tile
    uint32_t t_first, t_last, n_shared, n_seg, sk_tiles, cta, ctas;

    __host__ __device__ void init(const PrefillParams &p, uint32_t k_stages, uint32_t cta_, uint32_t ctas_) {
        ks = k_stages;
        cta = cta_;
        ctas = ctas_;
        sk_tiles = p.sk_tiles;
        if (p.split > 1) {  // (sk_tiles * split == ctas: a part lies in one tile)
            const uint64_t t0 = (uint64_t)(cta / p.split) * ks;
            u0 = t0 + part_begin(0, ks, cta % p.split, p.split);
            u1 = t0 + part_begin(0, ks, cta % p.split + 1, p.split);
        } else {
            u0 = part_begin(p.share_q, p.share_r, cta, ctas);
            u1 = part_begin(p.share_q, p.share_r, cta + 1, ctas);
        }
        n_shared = 0;
        t_first = t_last = 0;
        if (u1 > u0) {
            t_first = tile_of(u0);
            t_last = tile_of(u1 - 1);
            n_shared = t_last - t_first + 1;
        }
        n_seg = n_shared + p.dp_rounds;
    }
    __host__ __device__ uint32_t tile_of(uint64_t stage) const { return stage >> 32 ? (uint32_t)(stage / ks) : (uint32_t)stage / ks; }
    // Where part c of n begins, when each has q stages and r more are shared out (c r below 2^32): at a whole step of two
    // stages, if tiles consist of whole steps.
    __host__ __device__ uint64_t part_begin(uint64_t q, uint32_t r, uint32_t c, uint32_t n) const {
        const uint64_t u = q * c + r * c / n;
        return ks & 1u ? u : u & ~1ull;
    }
    __host__ __device__ void get(uint32_t j, uint32_t &tile, uint32_t &b, uint32_t &e) const {
        if (j < n_shared) {
            tile = t_last - j;
            const uint64_t t0 = (uint64_t)tile * ks;
            b = (uint32_t)((u0 > t0 ? u0 : t0) - t0);
            e = (uint32_t)((u1 < t0 + ks ? u1 : t0 + ks) - t0);
        } else {
            tile = sk_tiles + (j - n_shared) * ctas + cta;
            b = 0;
            e = ks;
        }
    }
};

// Activation rows the MMAs of a tile beginning at row m0 take: all BN, or for the last, ragged tile the rows there are,
// up to a multiple of 32 (each CTA brings half of them).  An MMA takes as long as it has columns: at 64 rows the step is then
// bound by the dequantisers.  (With single stages, all 256 columns and the rows that do not exist in the split tiles' sums -> without,
// 64 x 4096 x 4096 41 -> 32 us, 64 x 14336 x 4096 54 -> 43; 18.0 and 31.0 now.)
template <int BN>
__host__ __device__ __forceinline__ uint32_t tile_columns(uint32_t M, uint32_t m0) {
    const uint32_t left = M - m0;
    return left < BN ? (left + 31) / 32 * 32 : BN;
}

// ---- TMEM store (32 lanes x 32-bit, 32 consecutive columns) ------------------------------
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t (&a)[16],
                                          const uint32_t (&b)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,"
        "%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};"
        ::"r"(taddr), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]),
        "r"(a[7]), "r"(a[8]), "r"(a[9]), "r"(a[10]), "r"(a[11]), "r"(a[12]), "r"(a[13]), "r"(a[14]),
        "r"(a[15]), "r"(b[0]), "r"(b[1]), "r"(b[2]), "r"(b[3]), "r"(b[4]), "r"(b[5]), "r"(b[6]),
        "r"(b[7]), "r"(b[8]), "r"(b[9]), "r"(b[10]), "r"(b[11]), "r"(b[12]), "r"(b[13]), "r"(b[14]),
        "r"(b[15])
        : "memory");
}

// ---- nibble -> f16 expansion --------------------------------------------------------------
// One packed byte (two codes) indexes a 256-entry table of half2 {level[lo], level[hi]} in shared memory,
// replicated per lane (no bank conflicts; entries 256 bytes apart, half of that used): a permute, a load
// and the multiplication by the scale per two weights.  (Byte-permute lookups in registers take four times
// the instructions; the table's reads have room in the shared memory because a CTA of a pair moves half an
// activation tile per stage.)
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t level_pair(uint32_t word, int byte, uint32_t lane_word) {
    const uint32_t at = __byte_perm(word, lane_word, 0x7604u | ((uint32_t)byte << 4));  // {4 lane, the byte, 1, rank}
    uint32_t v;
    asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(at));
    return v;
}

// Half a stage of one weight row: 16 packed bytes -> 16 registers of f16x2.  `scale`: the block's, twice; PERK: where the pairs of
// scales of the sixteen pairs of k lie, the same for the whole warp.
template <bool PERK>
__device__ __forceinline__ void expand_half(const uint32_t *w, uint32_t scale, uint32_t lane_word, uint32_t (&out)[16]) {
    #pragma unroll
    for (int i = 0; i < 16; i += 4) {
        uint32_t s[4] = {scale, scale, scale, scale};
        if (PERK) asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(s[0]), "=r"(s[1]), "=r"(s[2]), "=r"(s[3]) : "r"(scale + i * 4u) : "memory");
        #pragma unroll
        for (int j = 0; j < 4; ++j) out[i + j] = hmul2(level_pair(w[i >> 2], j, lane_word), s[j]);
    }
}

// The sixteen f16 levels, for plain loads when the table is built (constant memory is read one index at a time).
__device__ const uint32_t g_level_f16[16] = {NF4_LEVEL_F16_BITS_LIST};

template <int BN, bool YF32, int SCALES>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
prefill_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_t,
               const __grid_constant__ CUtensorMap tmap_b, const __grid_constant__ CUtensorMap tmap_y,
               const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_ahead,
               const __grid_constant__ CUtensorMap tmap_s, const PrefillParams p) {
    using X = XRing<BN>;
    constexpr bool PERK = SCALES == kScalesPerK;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // In a cluster a CTA's shared-memory addresses carry its rank in the top byte: `own`.
    const uint32_t win = ptx::smem_addr(smem_raw), own = win & 0xff000000u;
    auto at = [&](uint32_t place) { return smem_raw + ((own | place) - win); };
    constexpr int kStageRows = kEpiBytes / (BM * (YF32 ? 4 : 2));  // activation rows per staging pass
    uint8_t *epi = at(kEpiAt);
    float *row_scales = reinterpret_cast<float *>(at(kRowScalesAt));  // BN factors of the tile's rows

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t rank = ptx::cluster_cta_rank(), pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    auto bar = [&](int i) { return (own | kBarsAt) + 8u * i; };

    const uint32_t k_stages = p.K / BK;
    // A tile's steps: two stages each (an odd last one has one), then one for each chunk of the adapter (T's hi and lo halves).
    WorkList wl;
    wl.init(p, k_stages, pair, pairs);

    if (p.split > 1) ptx::pdl_launch_dependents();  // the kernel that adds the parts: it waits for this one to complete
    if (win - own > kBarsAt) {  // (both CTAs alike) the places below are not ours
        if (threadIdx.x == 0) NF4_REPORT_FAILURE(g_prefill_error, g_prefill_error_host, 6);
        return;
    }
    // A step's codes (and scales) go to a slot of their ring; the L2 is asked for eight stages at a time, some twenty
    // ahead of their loads (weights that nobody has touched yet come from HBM).
    constexpr uint32_t kAhead = 3, kUnit = 8;  // requests to the L2 ahead, and stages of each
    auto ask_codes = [&](uint32_t ks, int32_t n0, const CodePlace &c) {
        const uint32_t full = bar(kBarCFull + c.full);
        ptx::mbar_arrive_expect_tx(full, kCodeTileBytes + (PERK ? kPerKBytes : SCALES == kScalesTma ? kScaleTileBytes : 0));
        ptx::tma_load_2d((own | kCodesAt) + c.slot * kCodeTileBytes, &tmap_w, (int32_t)(ks * (BK / 2)), n0, full);
        if (SCALES == kScalesTma)
            ptx::tma_load_2d(own | scales_place(c.slot), &tmap_s, (int32_t)(p.absmax ? ks & ~3u : ks & ~15u), n0, full);
        if (PERK) ptx::tma_load_2d(own | scales_place(c.slot), &tmap_s, (int32_t)(ks * BK), n0 / 64, full);
    };
    auto ask_l2 = [&](uint32_t ks, int32_t n0) { ptx::tma_prefetch_2d(&tmap_ahead, (int32_t)(ks * (BK / 2)), n0); };
    uint32_t asked = 0;  // steps of the first segment whose codes are on their way before anything else is in place
    if (warp == kCodeWarp) {
        uint32_t tile = 0, kb = 0, ke = 0;
        if (!PERK && wl.n_seg) wl.get(0, tile, kb, ke);
        asked = min((ke - kb + 1) / 2, (uint32_t)kCodeSlots);
        if (ptx::elect_one()) {
            for (int s = 0; s < 2 * kCodeSlots; ++s) ptx::mbar_init(bar(kBarCFull + s), 1);
            for (int s = 0; s < kCodeSlots; ++s) ptx::mbar_init(bar(kBarCEmpty + s), 8);   // the warps that dequantise a step
            ptx::fence_mbar_init();
            ptx::fence_proxy_async();
            const int32_t n0 = (int32_t)(((tile / p.m_tiles) * 2 + rank) * BM);
            for (uint32_t i = 0; i < asked; ++i) ask_codes(kb + 2 * i, n0, code_place(i));
            for (uint32_t k = kb; k < min(ke, kb + kAhead * kUnit); k += kUnit) ask_l2(k, n0);
        }
        __syncwarp();
    }
    if (threadIdx.x == 0) {
        for (int s = 0; s < kBarRing; ++s) {
            ptx::mbar_init(bar(kBarFull + s), 1 + kStepWarps);
            ptx::mbar_init(bar(kBarDone + s), 1);
        }
        ptx::mbar_init(bar(kBarAccFull), 1);
        ptx::mbar_init(bar(kBarAccEmpty), 16);      // the epilogue warps of both CTAs (used in the even one)
        ptx::fence_mbar_init();
        ptx::fence_proxy_async();
        ptx::prefetch_tmap(&tmap_x);
        ptx::prefetch_tmap(&tmap_y);
        if (p.lora_chunks) {
            ptx::prefetch_tmap(&tmap_t);
            ptx::prefetch_tmap(&tmap_b);
        }
    }
    // The scales of this group's next kDepth stages are in flight.  A position is walked, not divided out.
    constexpr int kDepth = 3;
    struct Pos {
        uint32_t seg, ks, ke;  // segment, stage in tile, the segment's end
        uint32_t before;       // steps before the segments after this one
        size_t row;            // index of the weight row's first scale
    } ahead{0, 0, 0, 0, 0};
    const uint32_t group = (warp - kFirstExpanderWarp) >> 2, odd = group >> 1, half = group & 1u;  // (of a dequantiser)
    const uint32_t q = warp & 3u, row_in_tile = q * 32 + lane;  // the TMEM lane quarter this warp may touch
    const uint32_t blocks_per_row = p.K / 64;
    auto enter = [&]() {  // the first main stage of this group in segment ahead.seg or a later one
        for (; ahead.seg < wl.n_seg; ++ahead.seg) {
            uint32_t tile, kb;
            wl.get(ahead.seg, tile, kb, ahead.ke);
            ahead.ks = kb + 2 * ((odd - ahead.before) & 1u) + half;
            ahead.before += (ahead.ke - kb + 1) / 2 + (ahead.ke == k_stages ? p.lora_chunks : 0);
            if (ahead.ks < ahead.ke) {
                // (rows beyond the last read its scales; nobody stores what comes of them)
                const uint32_t n0 = ((tile / p.m_tiles) * 2 + rank) * BM;
                ahead.row = (size_t)min(n0 + row_in_tile, p.N - 1) * blocks_per_row;
                return;
            }
        }
    };
    // The scale of the next stage as loaded: f32 bits or a u8 code.
    // Nothing is computed from it here: that would wait for the load, the latency the pipeline hides.
    auto fetch = [&]() -> uint32_t {
        if (SCALES != kScalesLoaded || ahead.seg >= wl.n_seg) return 0;
        const uint32_t v = p.absmax ? __float_as_uint(__ldg(p.absmax + ahead.row + ahead.ks)) : __ldg(p.scale_codes + ahead.row + ahead.ks);
        ahead.ks += kExpanderGroups;
        if (ahead.ks >= ahead.ke) {
            ++ahead.seg;
            enter();
        }
        return v;
    };
    uint32_t scales[kDepth] = {};
    const bool dequantiser = threadIdx.x >= kFirstExpanderWarp * 32 && threadIdx.x < kFirstEpilogueWarpB * 32;
    if (SCALES == kScalesLoaded && dequantiser) {
        enter();
        #pragma unroll
        for (int d = 0; d < kDepth; ++d) scales[d] = fetch();
    }
    // Block scales are used divided by a power of two (see weight_exponent)
    // ... and enter the product as f16: one multiplication from the loaded value.  (A u8 code's scale is
    // (code / 255) * scale of scales; dividing once instead of per code moves it by an ulp of f32.)
    float scale_unit = 1.0f;
    if (dequantiser) {
        // dequantiser (byte, half) writes sixteen lanes' copies, rotated so that a warp's stores spread over the banks
        const uint32_t i = threadIdx.x - kFirstExpanderWarp * 32, byte = i >> 1, half = i & 1u;
        const uint32_t e = __ldg(g_level_f16 + (byte & 15u)) | (__ldg(g_level_f16 + (byte >> 4)) << 16);
        if (!PERK) {
            const float w_down = ldexpf(1.0f, -weight_exponent(p.absmax, p.scale_codes, p.scale_of_scales));
            scale_unit = p.absmax ? w_down : __fdiv_rn(__ldg(p.scale_of_scales), 255.0f) * w_down;
        }
        #pragma unroll
        for (uint32_t q = 0; q < 4; ++q)
            *reinterpret_cast<uint4 *>(at(kTableAt) + byte * 256u + half * 64u + ((q + byte) & 3u) * 16u) = make_uint4(e, e, e, e);
    }
    if (warp == 1) {
        ptx::tmem_alloc_pair(own | kTmemSlotAt, kTmemCols);
        ptx::tmem_relinquish_pair();
    }
    // The barriers and the tensor memory of both CTAs are in place, and this CTA's table.
    ptx::tc_fence_before();
    __syncwarp();
    ptx::cluster_sync_all();
    ptx::tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<const uint32_t *>(at(kTmemSlotAt));
    const uint32_t tmem_acc = tmem_base;             // columns [0, 256)
    const uint32_t tmem_a = tmem_base + kAccCols;    // kASteps x 2 x 32 columns

    bool ok = true;
    auto step_done = [&](uint32_t step) { return ptx::mbar_wait_suspended(bar(kBarDone + step % kBarRing), (step / kBarRing) & 1u); };

    if (warp == 0) {
        // ============================ TMA producer ============================
        // The warp stays together and elects the thread that asks (see the issuer): a lane on its own in a branch took 300 to
        // 440 cycles a stage for its waits, arrivals and requests, which made this warp what every stage waited for.
        // The f16 activations and T come from the pre-pass, which may still be running: this
        // kernel is its programmatic dependent (the dequantisers start on the weights at once).
        ptx::pdl_wait();
        uint32_t step = 0, slot = 0;
        uint32_t user[X::kSlots];  // of the slots from the next one on: the last step that used it, plus one
        #pragma unroll
        for (uint32_t i = 0; i < X::kSlots; ++i) user[i] = 0;
        auto take = [&]() -> uint32_t {  // the next slot, once its last user is done
            if (user[0]) ok = step_done(user[0] - 1);
            #pragma unroll
            for (uint32_t i = 0; i + 1 < X::kSlots; ++i) user[i] = user[i + 1];
            user[X::kSlots - 1] = step + 1;
            const uint32_t at = own | X::place(slot);
            slot = X::next(slot);
            return at;
        };
        const uint32_t full0 = bar(kBarFull), pair_full0 = ptx::map_to_rank(full0, 0), tile_bytes = p.box_rows * (BK * 2);
        for (uint32_t seg = 0; seg < wl.n_seg && ok; ++seg) {
            uint32_t tile, kb, ke;
            wl.get(seg, tile, kb, ke);
            const uint32_t tile_m0 = (tile % p.m_tiles) * BN, n0 = ((tile / p.m_tiles) * 2 + rank) * BM;
            const uint32_t m0 = tile_m0 + rank * (tile_columns<BN>(p.M, tile_m0) / 2);  // (the box may be longer; the MMAs take what counts)
            for (uint32_t ks = kb; ks < ke && ok; ks += 2, ++step) {
                const uint32_t dst = take();
                if (!ok) break;
                const bool two = ks + 1 < ke;
                const uint32_t b = 8u * (step % kBarRing);
                if (ptx::elect_one()) {
                    if (rank == 0) ptx::mbar_arrive_expect_tx(full0 + b, (two ? 4u : 2u) * tile_bytes);
                    ptx::tma_load_2d_pair(dst, &tmap_x, (int32_t)(ks * BK), (int32_t)m0, pair_full0 + b);
                    if (two) ptx::tma_load_2d_pair(dst + X::kTile, &tmap_x, (int32_t)((ks + 1) * BK), (int32_t)m0, pair_full0 + b);
                }
                __syncwarp();
            }
            // the adapter's steps follow a tile's last main step: a slot for the 128 x 64 tile of LoRA B (ranks beyond the
            // adapter's read as zero), one for the halves of T
            for (uint32_t j = 0; ke == k_stages && j < p.lora_chunks && ok; ++j, ++step) {
                const uint32_t dst_b = take(), dst = ok ? take() : 0u;
                if (!ok) break;
                const uint32_t b = 8u * (step % kBarRing);
                if (ptx::elect_one()) {
                    if (rank == 0) ptx::mbar_arrive_expect_tx(full0 + b, 2 * (2 * tile_bytes + kLoraTileBytes));
                    ptx::tma_load_2d_pair(dst_b, &tmap_b, (int32_t)(j * BK), (int32_t)n0, pair_full0 + b);
                    ptx::tma_load_2d_pair(dst, &tmap_t, (int32_t)(j * BK), (int32_t)m0, pair_full0 + b);
                    ptx::tma_load_2d_pair(dst + X::kTile, &tmap_t, (int32_t)((p.lora_chunks + j) * BK), (int32_t)m0, pair_full0 + b);
                }
                __syncwarp();
            }
        }
        if (!ok && lane == 0) NF4_REPORT_FAILURE(g_prefill_error, g_prefill_error_host, 1);
    } else if (warp == 1) {
        // ============================= MMA issuer =============================
        // One thread of the even CTA issues the pair's MMAs: per step one wait, eight MMAs, one commit.  The
        // warp stays together and elects the thread where it issues, so that addresses and descriptors are
        // uniform registers; one lane on its own in a branch spent 77 cycles on each MMA, which takes 128.
        if (rank == 0) {
            uint32_t step = 0, slot = 0;
            auto step_full = [&]() { return ptx::mbar_wait_suspended(bar(kBarFull + step % kBarRing), (step / kBarRing) & 1u); };
            for (uint32_t seg = 0; seg < wl.n_seg && ok; ++seg) {
                uint32_t tile, kb, ke;
                wl.get(seg, tile, kb, ke);
                const uint32_t columns = tile_columns<BN>(p.M, (tile % p.m_tiles) * BN);
                const uint32_t idesc_main = ptx::f16_idesc(0, 2 * BM, columns, false, false);  // f16 x f16
                const uint32_t idesc_lora = ptx::f16_idesc(1, 2 * BM, columns, false, false);  // bf16 x bf16
                // the epilogues must have read the previous segment out of the accumulators
                ok = ptx::mbar_wait_suspended(bar(kBarAccEmpty), (seg & 1u) ^ 1u);
                for (uint32_t ks = kb; ks < ke && ok; ks += 2, ++step, slot = X::next(slot)) {
                    const uint64_t bdesc = ptx::sw128_desc(X::place(slot));
                    const uint32_t a_cols = tmem_a + step % kASteps * (2 * kStageCols);
                    ok = step_full();
                    if (!ok) break;
                    ptx::tc_fence_after();
                    if (ptx::elect_one()) {
                        // 16 k = 8 TMEM columns of the weight stage = 32 bytes inside the
                        // activation tile's swizzled row (+2 in the encoded address)
                        ptx::mma_ts_f16_pair(tmem_acc, a_cols, bdesc, idesc_main, ks != kb ? 1u : 0u);
                        #pragma unroll
                        for (uint32_t i = 1; i < 4; ++i) ptx::mma_ts_f16_pair(tmem_acc, a_cols + 8 * i, bdesc + 2 * i, idesc_main, 1u);
                        if (ks + 1 < ke) {
                            #pragma unroll
                            for (uint32_t i = 0; i < 4; ++i)
                                ptx::mma_ts_f16_pair(tmem_acc, a_cols + kStageCols + 8 * i, bdesc + (X::kTile >> 4) + 2 * i, idesc_main, 1u);
                        }
                        ptx::tc_commit_pair(bar(kBarDone + step % kBarRing));
                    }
                    __syncwarp();
                }
                for (uint32_t j = 0; ke == k_stages && j < p.lora_chunks && ok; ++j, ++step) {
                    const uint32_t left = p.rank - j * 64, nk16 = ((left < 64 ? left : 64) + 15) / 16;
                    const uint64_t adesc = ptx::sw128_desc(X::place(slot));
                    slot = X::next(slot);
                    const uint64_t bdesc = ptx::sw128_desc(X::place(slot));
                    slot = X::next(slot);
                    ok = step_full();
                    if (!ok) break;
                    ptx::tc_fence_after();
                    if (ptx::elect_one()) {
                        for (uint32_t i = 0; i < nk16; ++i) ptx::mma_ss_f16_pair(tmem_acc, adesc + 2 * i, bdesc + 2 * i, idesc_lora, 1u);
                        for (uint32_t i = 0; i < nk16; ++i)
                            ptx::mma_ss_f16_pair(tmem_acc, adesc + 2 * i, bdesc + (X::kTile >> 4) + 2 * i, idesc_lora, 1u);
                        ptx::tc_commit_pair(bar(kBarDone + step % kBarRing));
                    }
                    __syncwarp();
                }
                if (ok && ptx::elect_one()) ptx::tc_commit_pair(bar(kBarAccFull));
                __syncwarp();
            }
            if (!ok && lane == 0) NF4_REPORT_FAILURE(g_prefill_error, g_prefill_error_host, 2);
        }
    } else if (warp < 6 || warp >= kFirstEpilogueWarpB) {
        // ============================== epilogue ==============================
        // The MMAs of the next tile wait for the accumulator, so it is read out as fast as eight
        // warps can (two per TMEM lane quarter, each taking half of the columns): half of the tile
        // (bf16) or a quarter of it (f32) goes through one staging buffer at a time, and the accumulator is
        // handed back before the last values are stored; their TMA store then overlaps the next tile's MMAs.
        const uint32_t set = warp >= kFirstEpilogueWarpB ? 1u : 0u;
        const uint32_t epi_thread = set * 128 + (warp - (set ? kFirstEpilogueWarpB : 2)) * 32 + lane;
        const uint32_t epi_leader = (warp == 2 && lane == 0);
        const uint32_t acc_lane = tmem_acc + ((q * 32) << 16);
        // this warp's eight 16-column TMEM loads of a tile: within every staging pass the first
        // set takes the first half of the pass's activation rows, the second set the other half
        constexpr uint32_t kHalfRows = kStageRows / 2, kPerPass = kHalfRows / 16;
        constexpr uint32_t kLoads = BN / 2 / 16;
        auto col_of = [&](uint32_t k) {
            return (k / kPerPass) * kStageRows + set * kHalfRows + (k % kPerPass) * 16;
        };
        const uint32_t acc_empty = ptx::map_to_rank(bar(kBarAccEmpty), 0);
        ptx::pdl_wait();  // the rows' factors come from the pre-pass, which also cleared the flags
        float *own_partial = p.partial + (size_t)blockIdx.x * (BM * BN) + row_in_tile;
        for (uint32_t seg = 0; seg < wl.n_seg && ok; ++seg) {
            const uint32_t i = seg;  // the accumulator's barriers alternate per segment
            const bool more = seg + 1 < wl.n_seg;  // (what nobody waits for must not be under way when the other CTA ends)
            uint32_t tile, kb, ke;
            wl.get(seg, tile, kb, ke);
            const uint32_t n0 = ((tile / p.m_tiles) * 2 + rank) * BM, m0 = (tile % p.m_tiles) * BN;
            const uint32_t n = n0 + row_in_tile;
            if (ke != k_stages || p.split > 1) {
                // The leading stages of a tile that a neighbour finishes, or a part of one: the raw sums go to this
                // CTA's place in global memory ([activation row][weight row]: a warp's stores are
                // whole lines; a thread's values 64 bytes in a row were measured 15 % slower over
                // the whole GEMM), then the flag goes up.
                ok = ptx::mbar_wait_suspended(bar(kBarAccFull), i & 1u);
                if (!ok) break;
                ptx::tc_fence_after();
                uint32_t v[16];
                for (uint32_t k = 0; k < kLoads; ++k) {
                    if (m0 + col_of(k) >= p.M) continue;  // rows that do not exist
                    ptx::tmem_ld16(acc_lane + col_of(k), v);
                    ptx::tmem_wait_ld();
                    float *dst = own_partial + (size_t)col_of(k) * BM;
                    #pragma unroll
                    for (int r = 0; r < 16; ++r) dst[r * BM] = __uint_as_float(v[r]);
                }
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0 && more) ptx::mbar_arrive_cluster(acc_empty);
                asm volatile("bar.sync 1, 256;" ::: "memory");
                if (epi_leader && p.split <= 1) {
                    __threadfence();
                    atomicExch(p.sk_flags + blockIdx.x, 1u);
                }
                continue;
            }
            // a tile whose leading stages other pairs multiplied: the pairs before this one, back to
            // the one that began the tile; a CTA's helpers have its own rank
            uint32_t first_helper = pair;
            if (kb != 0) {
                const uint64_t t0 = (uint64_t)tile * k_stages;
                do {
                    --first_helper;
                } while (first_helper > 0 && wl.part_begin(p.share_q, p.share_r, first_helper, pairs) > t0);
            }
            // the rows' factors go to shared memory while the MMAs still run: a global load per
            // value inside the read-out would wait for L2 every time (the L1 left beside 227 KB
            // of shared memory is small and the dequantisers stream through it)
            if (epi_thread < BN) row_scales[epi_thread] = m0 + epi_thread < p.M ? __ldg(p.row_scale + m0 + epi_thread) : 1.0f;
            ok = ptx::mbar_wait_suspended(bar(kBarAccFull), i & 1u);
            if (!ok) break;
            ptx::tc_fence_after();
            if (first_helper != pair && epi_leader) {
                // bounded wait for the helpers' flags (they dumped before anything else they did)
                const uint64_t t_begin = ptx::global_timer_ns();
                for (uint32_t h = first_helper; h < pair && ok; ++h) {
                    while (ptx::ld_acquire_gpu_u32(p.sk_flags + 2 * h + rank) == 0u) {
                        if (ptx::global_timer_ns() - t_begin > (uint64_t)p.wait_ns) {
                            ok = false;
                            break;
                        }
                        __nanosleep(64);
                    }
                }
                if (!ok) NF4_REPORT_FAILURE(g_prefill_error, g_prefill_error_host, 5);  // the sums are wrong; the flag says so
                ok = true;  // the read-out goes on (every role must finish its segments)
            }
            if constexpr (YF32) {
                const float bias = (p.bias && n < p.N) ? __ldg(p.bias + n) : 0.0f;
                uint32_t va[16], vb[16];
                ptx::tmem_ld16(acc_lane + col_of(0), va);
                // staging layout: [kStageRows activation rows][BM weight rows]
                auto stage_chunk = [&](const uint32_t (&v)[16], uint32_t col) {
                    const uint32_t r0 = col % kStageRows;
                    // the factors first, as vectors: a load per value between the stores could not be
                    // moved ahead of them (both are shared memory) and each would wait out its latency
                    float rs[16];
                    #pragma unroll
                    for (int r4 = 0; r4 < 4; ++r4) {
                        const float4 f4 = reinterpret_cast<const float4 *>(row_scales + col)[r4];
                        rs[4 * r4 + 0] = f4.x;
                        rs[4 * r4 + 1] = f4.y;
                        rs[4 * r4 + 2] = f4.z;
                        rs[4 * r4 + 3] = f4.w;
                    }
                    #pragma unroll
                    for (int r = 0; r < 16; ++r) {
                        const float f = fmaf(__uint_as_float(v[r]), rs[r], bias);
                        reinterpret_cast<float *>(epi)[(r0 + r) * BM + row_in_tile] = f;
                    }
                };
                auto add_helpers = [&](uint32_t (&v)[16], uint32_t col) {
                    if (m0 + col >= p.M) return;
                    for (uint32_t h = first_helper; h < pair; ++h) {
                        const float *src = p.partial + (size_t)(2 * h + rank) * (BM * BN) + (size_t)col * BM + row_in_tile;
                        float part[16];
                        #pragma unroll
                        for (int r = 0; r < 16; ++r) part[r] = __ldcg(src + r * BM);
                        #pragma unroll
                        for (int r = 0; r < 16; ++r) v[r] = __float_as_uint(__uint_as_float(v[r]) + part[r]);
                    }
                };
                for (uint32_t k = 0; k < kLoads; k += 2) {
                    if (k % kPerPass == 0) {
                        // the TMA store that last read the staging buffer must be done with it
                        if (epi_leader) ptx::tma_store_wait_read<0>();
                        asm volatile("bar.sync 1, 256;" ::: "memory");
                    }
                    ptx::tmem_wait_ld();
                    ptx::tmem_ld16(acc_lane + col_of(k + 1), vb);
                    if (first_helper != pair) add_helpers(va, col_of(k));
                    stage_chunk(va, col_of(k));
                    ptx::tmem_wait_ld();
                    if (first_helper != pair) add_helpers(vb, col_of(k + 1));
                    if (k + 2 < kLoads) {
                        ptx::tmem_ld16(acc_lane + col_of(k + 2), va);
                    } else {
                        // this warp's part of the accumulator is read: hand it back to the MMA threads
                        ptx::tc_fence_before();
                        __syncwarp();
                        if (lane == 0 && more) ptx::mbar_arrive_cluster(acc_empty);
                    }
                    stage_chunk(vb, col_of(k + 1));
                    if ((k + 2) % kPerPass == 0) {
                        ptx::fence_proxy_async();
                        asm volatile("bar.sync 1, 256;" ::: "memory");
                        // (an odd number of 128-row tiles: the last odd CTA's rows do not exist)
                        const uint32_t m = m0 + (k / kPerPass) * kStageRows;
                        if (p.y_ragged && n0 + BM > p.N) {
                            #pragma unroll 1
                            for (uint32_t e = epi_thread; e < kStageRows * BM; e += 256) {
                                const uint32_t row = m + e / BM, col = n0 + e % BM;
                                if (row < p.M && col < p.N) static_cast<float *>(p.y_ragged)[row * p.ldy + col] = reinterpret_cast<const float *>(epi)[e];
                            }
                        } else if (epi_leader && n0 < p.N && m < p.M) {
                            ptx::tma_store_2d(&tmap_y, own | kEpiAt, (int32_t)n0, (int32_t)m);
                            ptx::tma_store_commit();
                        }
                    }
                }
            } else {
                // bf16: fragments of 16 weight rows x 32 columns, so that two neighbouring columns are converted to one
                // register and a transposing matrix store puts eight weight rows of a column side by side: 16 two-byte
                // stores for 16 columns took 400 cycles (700 x 4096 x 14336: 89.4 -> 86.8 us, 1000 x 8192 x 8192 129 -> 126,
                // 2048 x 4096 x 14336, at the power limit, 209 -> 206).  The first half of the columns goes to the staging
                // buffer and out; half of the second is in registers when the buffer is free again.
                const uint32_t fn = lane >> 2, fm = 2u * (lane & 3u), mi = lane & 7u, mq = lane >> 3;
                const uint32_t nq = n0 + q * 32 + fn;
                auto bias_of = [&](uint32_t row) { return p.bias && row < p.N ? __ldg(p.bias + row) : 0.0f; };
                auto convert = [&](uint32_t col, uint32_t half, uint32_t *w) {  // -> eight registers
                    uint32_t v[16];
                    ptx::tmem_ld_fragments(acc_lane + ((half * 16) << 16) + col, v);
                    const float b0 = bias_of(nq + half * 16), b1 = bias_of(nq + half * 16 + 8);
                    ptx::tmem_wait_ld();
                    if (m0 + col < p.M)
                        for (uint32_t h = first_helper; h < pair; ++h) {
                            const float *src = p.partial + (size_t)(2 * h + rank) * (BM * BN) + (size_t)(col + fm) * BM + q * 32 + half * 16 + fn;
                            #pragma unroll
                            for (int j = 0; j < 4; j += 2) {
                                float part[8];
                                #pragma unroll
                                for (int r = 0; r < 8; ++r) part[r] = __ldcg(src + (8 * (j + (r >> 2)) + (r & 1)) * BM + ((r >> 1) & 1) * 8);
                                #pragma unroll
                                for (int r = 0; r < 8; ++r) v[4 * j + r] = __float_as_uint(__uint_as_float(v[4 * j + r]) + part[r]);
                            }
                        }
                    #pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float2 rs = *reinterpret_cast<const float2 *>(row_scales + col + 8 * j + fm);
                        #pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            const __nv_bfloat162 o = __floats2bfloat162_rn(fmaf(__uint_as_float(v[4 * j + 2 * r]), rs.x, r ? b1 : b0),
                                                                          fmaf(__uint_as_float(v[4 * j + 2 * r + 1]), rs.y, r ? b1 : b0));
                            w[2 * j + r] = *reinterpret_cast<const uint32_t *>(&o);
                        }
                    }
                };
                // staging: two boxes of 64 weight rows, [128 activation rows][128 bytes] with the store's swizzle
                auto stage = [&](uint32_t col, uint32_t half, const uint32_t *w) {
                    const uint32_t oct = q * 4 + half * 2 + (mq & 1u);
                    #pragma unroll
                    for (uint32_t j = 0; j < 4; j += 2) {
                        const uint32_t row = col + (j + (mq >> 1)) * 8 + mi;
                        ptx::stmatrix_x4_trans((own | kEpiAt) + (oct >> 3) * (kEpiBytes / 2) + row * 128 + (((oct & 7u) ^ (row & 7u)) << 4),
                                               w[2 * j], w[2 * j + 1], w[2 * j + 2], w[2 * j + 3]);
                    }
                };
                auto send = [&](uint32_t m) {  // the staged 128 activation rows from m on (an odd last CTA has no weight rows)
                    ptx::fence_proxy_async();
                    asm volatile("bar.sync 1, 256;" ::: "memory");
                    if (p.y_ragged && n0 + BM > p.N) {
                        #pragma unroll 1
                        for (uint32_t e = epi_thread; e < kStageRows * BM; e += 256) {
                            const uint32_t r = e / BM, c = e % BM;
                            if (m + r < p.M && n0 + c < p.N)
                                static_cast<__nv_bfloat16 *>(p.y_ragged)[(size_t)(m + r) * p.ldy + n0 + c] = *reinterpret_cast<const __nv_bfloat16 *>(
                                    epi + (c >> 6) * (kEpiBytes / 2) + r * 128 + ((((c >> 3) & 7u) ^ (r & 7u)) << 4) + (c & 7u) * 2);
                        }
                    } else if (epi_leader) {
                        if (n0 < p.N) ptx::tma_store_2d(&tmap_y, own | kEpiAt, (int32_t)n0, (int32_t)m);
                        if (n0 + 64 < p.N) ptx::tma_store_2d(&tmap_y, (own | kEpiAt) + kEpiBytes / 2, (int32_t)n0 + 64, (int32_t)m);
                        ptx::tma_store_commit();
                    }
                };
                auto buffer_free = [&]() {
                    if (epi_leader) ptx::tma_store_wait_read<0>();
                    asm volatile("bar.sync 1, 256;" ::: "memory");
                };
                auto hand_back = [&]() {  // this warp's part of the accumulator is read
                    ptx::tc_fence_before();
                    __syncwarp();
                    if (lane == 0 && more) ptx::mbar_arrive_cluster(acc_empty);
                };
                const uint32_t at = set * 64;  // a set's columns of a half: four pieces of 16 weight rows x 32 columns
                uint32_t w[2][8];
                buffer_free();
                #pragma unroll
                for (uint32_t c = 0; c < 4; ++c) {
                    convert(at + (c >> 1) * 32, c & 1u, w[0]);
                    stage(at + (c >> 1) * 32, c & 1u, w[0]);
                }
                send(m0);
                if (BN > kStageRows && m0 + kStageRows < p.M) {
                    #pragma unroll
                    for (uint32_t c = 0; c < 2; ++c) convert(kStageRows + at, c, w[c]);
                    buffer_free();
                    #pragma unroll
                    for (uint32_t c = 0; c < 2; ++c) stage(at, c, w[c]);
                    #pragma unroll
                    for (uint32_t c = 0; c < 2; ++c) {
                        convert(kStageRows + at + 32, c, w[0]);
                        if (c == 1) hand_back();
                        stage(at + 32, c, w[0]);
                    }
                    send(m0 + kStageRows);
                } else {
                    hand_back();
                }
            }
        }
        if (epi_leader) ptx::tma_store_wait_read<0>();  // (what was read is on its way; the kernel's end waits for it)
        if (!ok && lane == 0) NF4_REPORT_FAILURE(g_prefill_error, g_prefill_error_host, 3);
    } else if (warp >= kFirstExpanderWarp && warp < kFirstEpilogueWarpB) {
        // ============================ dequantisers ============================
        // Four groups of four warps; groups 0 and 1 take the two stages of the even steps (counted over this CTA's tiles),
        // groups 2 and 3 those of the odd ones.
        // Within a group the warp's number modulo 4 names the TMEM lane quarter it may write, and
        // the lane the weight row: 32 packed bytes + the scale in, 64 f16 values out, stored as
        // 32 TMEM columns (two f16 per cell, even k in the low half) of the stage's place in the ring.
        const uint32_t lane_word = lane * 4u | kTableAt | own;  // bytes {4 lane, 0, 1, rank}: see level_pair
        const uint32_t lane_base = tmem_a + ((q * 32) << 16);

        // A group has every other step, the adapter's and the missing half of an odd last one included (nothing to write
        // there, but its turn on the barriers): then it is never two rounds of Done ahead, where a parity would be the wrong
        // round's, nor of the codes' barriers (see code_place).
        uint32_t before = 0, blocks = 0;  // steps, and main ones, before the segment
        const uint32_t swizzle = (row_in_tile >> 1) & 3u, row_at = (own | kCodesAt) + row_in_tile * 64u;
        const uint32_t chunk0 = row_at + (((half * 2) ^ swizzle) << 4), chunk1 = row_at + (((half * 2 + 1) ^ swizzle) << 4);
        const uint32_t full0 = ptx::map_to_rank(bar(kBarFull), 0);
        auto columns_free = [&](uint32_t step) { return step < kASteps || step_done(step - kASteps); };
        auto nothing = [&](uint32_t step) {
            ok = columns_free(step);
            __syncwarp();
            if (ok && lane == 0) ptx::mbar_arrive_cluster(full0 + 8u * (step % kBarRing));
        };
        for (uint32_t seg = 0; seg < wl.n_seg && ok; ++seg) {
            uint32_t tile, kb, ke;
            wl.get(seg, tile, kb, ke);
            const uint32_t steps = (ke - kb + 1) / 2;
            for (uint32_t j = (odd - before) & 1u; j < steps && ok; j += 2) {
                const uint32_t step = before + j;
                const CodePlace c = code_place(blocks + j);
                const uint32_t slot = c.slot;
                if (!ptx::mbar_wait_suspended(bar(kBarCFull + c.full), c.parity)) {
                    ok = false;
                    break;
                }
                if (kb + 2 * j + half >= ke) {  // an odd last step's second half
                    if (lane == 0) ptx::mbar_arrive(bar(kBarCEmpty + slot));
                    nothing(step);
                    continue;
                }
                uint32_t w[8];
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                             : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(chunk0 + slot * kCodeTileBytes) : "memory");
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                             : "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7]) : "r"(chunk1 + slot * kCodeTileBytes) : "memory");
                uint32_t scale2 = scales[0];
                if constexpr (SCALES == kScalesTma) {
                    const uint32_t ks = kb + 2 * j + half, at = (own | scales_place(slot)) + row_in_tile * 16u;
                    if (p.absmax) asm volatile("ld.shared.u32 %0, [%1];" : "=r"(scale2) : "r"(at + (ks & 3u) * 4u) : "memory");
                    else asm volatile("ld.shared.u8 %0, [%1];" : "=r"(scale2) : "r"(at + (ks & 15u)) : "memory");
                }
                if constexpr (PERK) scale2 = (own | scales_place(slot)) + (q >> 1) * (2 * BK * 2) + half * (BK * 2);
                if constexpr (!PERK) {
                    const __half2 h = __float2half2_rn((p.absmax ? __uint_as_float(scale2) : (float)scale2) * scale_unit);
                    scale2 = *reinterpret_cast<const uint32_t *>(&h);
                }
                if constexpr (SCALES == kScalesLoaded) {
                    #pragma unroll
                    for (int d = 0; d + 1 < kDepth; ++d) scales[d] = scales[d + 1];
                    scales[kDepth - 1] = fetch();
                }
                uint32_t lo[16], hi[16];
                expand_half<PERK>(w, scale2, lane_word, lo);
                expand_half<PERK>(w + 4, scale2 + (PERK ? BK : 0), lane_word, hi);
                if (!columns_free(step)) {
                    ok = false;
                    break;
                }
                ptx::tc_fence_after();
                tmem_st32(lane_base + (step % kASteps * 2 + half) * kStageCols, lo, hi);
                ptx::tmem_wait_st();
                ptx::tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    ptx::mbar_arrive_cluster(full0 + 8u * (step % kBarRing));
                    // The slot goes back now that what was read from it has been used.  Right after the loads
                    // were issued is too early: the next copy, of another proxy, was seen to overtake them.
                    ptx::mbar_arrive(bar(kBarCEmpty + slot));
                }
            }
            before += steps;
            blocks += steps;
            if (ke != k_stages) continue;
            for (uint32_t j = (odd - before) & 1u; j < p.lora_chunks && ok; j += 2) nothing(before + j);
            before += p.lora_chunks;
        }
        if (!ok && lane == 0) NF4_REPORT_FAILURE(g_prefill_error, g_prefill_error_host, 4);
    }

    if (warp == kCodeWarp) {
        // ========================= packed codes =========================
        if (PERK) ptx::pdl_wait();
        uint32_t block = asked;
        for (uint32_t seg = 0; seg < wl.n_seg && ok; ++seg) {
            uint32_t tile, kb, ke;
            wl.get(seg, tile, kb, ke);
            const int32_t n0 = (int32_t)(((tile / p.m_tiles) * 2 + rank) * BM);
            if ((PERK || seg) && ptx::elect_one())
                for (uint32_t k = kb; k < min(ke, kb + kAhead * kUnit); k += kUnit) ask_l2(k, n0);
            __syncwarp();
            for (uint32_t ks = kb; ks < ke; ks += 2) {
                const uint32_t ahead = ks + kAhead * kUnit;
                const bool to_l2 = (ks - kb) % kUnit == 0 && ahead < ke;
                if (seg == 0 && ks < kb + 2 * asked) {
                    if (to_l2 && ptx::elect_one()) ask_l2(ahead, n0);
                    __syncwarp();
                    continue;
                }
                // (every block in turn: a round of the slot's Empty is never passed by)
                const CodePlace c = code_place(block);
                ok = ptx::mbar_wait_suspended(bar(kBarCEmpty + c.slot), (block / kCodeSlots & 1u) ^ 1u);
                if (!ok) break;
                if (ptx::elect_one()) {
                    ask_codes(ks, n0, c);
                    if (to_l2) ask_l2(ahead, n0);
                }
                __syncwarp();
                ++block;
            }
        }
        if (!ok && lane == 0) NF4_REPORT_FAILURE(g_prefill_error, g_prefill_error_host, 7);
    }

    if (!ok) ptx::let_flights_land();
    __syncwarp();
    // neither CTA leaves, or gives its tensor memory back, while the other may still signal it
    ptx::tc_fence_before();
    ptx::cluster_sync_all();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc_pair(tmem_base, kTmemCols);
    }
}

// ---- the sums of a tile whose stages several pairs shared --------------------------------------------------
// y[m][n] = (sum over the parts, in order, of partial[part][m][n]) * row factor + bias.  A warp takes one activation row of a
// CTA's 128 weight rows, a lane four of them.  One pair that collected the others' sums in its read-out, a helper and
// sixteen columns at a time, took 10 us (300 x 3584 x 3584), 14 (512 x 4096 x 4096, f32) and 23 (99 x 20288 x 512, twelve
// helpers); a launch of its own has all SMs' loads in flight, and no CTA waits for another one.
template <int BN, bool YF32>
__global__ void __launch_bounds__(256)
sum_parts_kernel(const float *__restrict__ partial, uint32_t split, uint32_t m_tiles, uint32_t M, uint32_t N, const float *__restrict__ row_scale,
                 const float *__restrict__ bias, void *__restrict__ y, uint64_t ldy) {
    ptx::pdl_wait();
    const uint32_t lane = threadIdx.x & 31u, col = blockIdx.x * 8 + (threadIdx.x >> 5);  // of the tile's activation rows
    const uint32_t tile = blockIdx.y >> 1, rank = blockIdx.y & 1u;
    const uint32_t m = tile % m_tiles * BN + col, n = (tile / m_tiles * 2 + rank) * BM + lane * 4;
    if (m >= M || n >= N) return;
    const float4 *src = reinterpret_cast<const float4 *>(partial + ((size_t)(tile * split * 2 + rank) * BN + col) * BM) + lane;
    constexpr size_t kPart = 2 * (size_t)BN * BM / 4;  // a pair's parts, in float4
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    constexpr uint32_t kInFlight = 8;
    for (uint32_t s = 0; s < split; s += kInFlight) {
        float4 p[kInFlight];
        #pragma unroll
        for (uint32_t i = 0; i < kInFlight; ++i)
            p[i] = s + i < split ? __ldcg(src + (s + i) * kPart) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        #pragma unroll
        for (uint32_t i = 0; i < kInFlight; ++i) {
            if (s + i >= split) break;
            v.x += p[i].x;
            v.y += p[i].y;
            v.z += p[i].z;
            v.w += p[i].w;
        }
    }
    const float rs = __ldg(row_scale + m);
    float o[4] = {v.x, v.y, v.z, v.w};
    #pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = fmaf(o[i], rs, bias && n + i < N ? __ldg(bias + n + i) : 0.0f);
    const size_t at = (size_t)m * ldy + n;
    if (n + 3 < N) {  // (rows and n are whole 16-byte pieces of f32, 8-byte ones of bf16)
        if (YF32) {
            *reinterpret_cast<float4 *>(static_cast<float *>(y) + at) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
            const __nv_bfloat162 a = __floats2bfloat162_rn(o[0], o[1]), b = __floats2bfloat162_rn(o[2], o[3]);
            *reinterpret_cast<uint2 *>(static_cast<__nv_bfloat16 *>(y) + at) =
                make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
        }
        return;
    }
    #pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (n + i >= N) break;
        if (YF32) static_cast<float *>(y)[at + i] = o[i];
        else static_cast<__nv_bfloat16 *>(y)[at + i] = __float2bfloat16_rn(o[i]);
    }
}

// ---- weights in the other orientation: repacking before the GEMM ---------------------------
// W [d_in][d_out] with the 64-blocks along d_out (the reference's Burn layout) is brought into the
// form the GEMM's dequantisers read: codes_t[n][k / 2] (the same nibbles, transposed, so exact) and
// scales_t[n / 64][k] (f16 of scale / 2^e, the rounding the GEMM applies to a scale anyway).

struct RepackParams {
    const uint8_t *codes;
    const float *absmax;
    const uint8_t *scale_codes;
    const float *scale_of_scales;
    const void *b;              // adapter factor B [r][N], or null
    uint8_t *codes_t;
    __half *scales_t;
    __nv_bfloat16 *b_t;
    uint32_t K, N, r;
    int32_t factor_out_in;      // the factor comes as [N][r]
    uint32_t code_cols, code_blocks;              // CTAs of the nibbles: tiles of 128 n x 256 k
    uint32_t scale_cols, scale_blocks;            // CTAs of the scales: 32 x 32 tiles
    uint32_t adapter_blocks;                      // CTAs of the factor: 32 x 32 tiles
};

// Nibbles.  A CTA turns 256 k x 128 n.  A thread takes eight words (8 k x 8 n) straight from global memory, all
// loads of its two blocks in flight, transposes each in registers (halves and bytes by permutes, nibbles by masks: 32
// operations for 32 bytes) and leaves the words in shared memory, from where whole 128-byte lines go out.  Bound by the
// bytes; picking nibbles out of shared memory byte by byte, into 8-byte pieces of lines, took 33 us for 4096 x 14336 with its
// scales and factors; now 15.
__device__ __forceinline__ void transpose_nibbles(uint32_t (&w)[8]) {  // nibble c of word j <-> nibble j of word c
    uint32_t h[8], b[8];
    #pragma unroll
    for (int j = 0; j < 4; ++j) {
        h[j] = __byte_perm(w[j], w[j + 4], 0x5410);      // columns 0-3 of rows j, j + 4
        h[j + 4] = __byte_perm(w[j], w[j + 4], 0x7632);  // columns 4-7
    }
    #pragma unroll
    for (int c = 0; c < 8; c += 4) {
        #pragma unroll
        for (int j = 0; j < 2; ++j) {
            b[c + j] = __byte_perm(h[c + j], h[c + j + 2], 0x6240);      // columns c, c + 1 of rows j, j + 2, j + 4, j + 6
            b[c + j + 2] = __byte_perm(h[c + j], h[c + j + 2], 0x7351);  // columns c + 2, c + 3
        }
    }
    #pragma unroll
    for (int c = 0; c < 8; c += 2) {
        w[c] = (b[c] & 0x0f0f0f0fu) | ((b[c + 1] << 4) & 0xf0f0f0f0u);
        w[c + 1] = ((b[c] >> 4) & 0x0f0f0f0fu) | (b[c + 1] & 0xf0f0f0f0u);
    }
}

__device__ __forceinline__ void repack_codes_block(const RepackParams &p, uint32_t block, uint32_t *tile) {
    const uint32_t n0 = (block % p.code_cols) * 128, k0 = (block / p.code_cols) * 256, t = threadIdx.x;
    const uint32_t j = t & 15u, i0 = t >> 4;  // eight columns n0 + 8 j; eight rows k0 + 8 i, i = i0 and i0 + 16
    const uint8_t *src = p.codes + (size_t)k0 * (p.N / 2) + n0 / 2 + j * 4;
    uint32_t w[2][8];
    #pragma unroll
    for (uint32_t u = 0; u < 2; ++u) {
        const uint32_t i = i0 + u * 16;
        const bool in = n0 + j * 8 < p.N && k0 + i * 8 < p.K;  // (both are multiples of 64)
        #pragma unroll
        for (uint32_t q = 0; q < 8; ++q)
            w[u][q] = in ? __ldg(reinterpret_cast<const uint32_t *>(src + (size_t)(i * 8 + q) * (p.N / 2))) : 0u;
    }
    // tile[n][i ^ 2 (n / 8)]: a warp's stores (sixteen j, two i) and its loads of pairs hit all banks
    #pragma unroll
    for (uint32_t u = 0; u < 2; ++u) {
        transpose_nibbles(w[u]);
        #pragma unroll
        for (uint32_t c = 0; c < 8; ++c) tile[(j * 8 + c) * 32 + ((i0 + u * 16) ^ (2 * j))] = w[u][c];
    }
    __syncthreads();
    const uint32_t pair = t & 15u;
    if (k0 + pair * 16 >= p.K) return;
    uint8_t *dst = p.codes_t + (size_t)n0 * (p.K / 2) + k0 / 2 + pair * 8;
    #pragma unroll
    for (uint32_t n = t >> 4; n < 128; n += 16) {
        if (n0 + n >= p.N) break;
        const uint2 v = *reinterpret_cast<const uint2 *>(tile + n * 32 + ((2 * pair) ^ (2 * (n >> 3))));
        *reinterpret_cast<uint2 *>(dst + (size_t)n * (p.K / 2)) = v;
    }
}

// scales_t[b][k] = f16(scale(k, b) / 2^e), scale(k, b) the scale of block k * (N / 64) + b.
__device__ __forceinline__ void repack_scales_block(const RepackParams &p, uint32_t block, float (*tile)[33]) {
    const uint32_t blocks_per_row = p.N / 64;
    const int w_exp = weight_exponent(p.absmax, p.scale_codes, p.scale_of_scales);
    const float w_down = ldexpf(1.0f, -w_exp);
    const float sos = p.scale_codes ? __ldg(p.scale_of_scales) : 0.0f;
    const uint32_t b0 = (block % p.scale_cols) * 32, k0 = (block / p.scale_cols) * 32;
    const uint32_t tx = threadIdx.x & 31u, ty = threadIdx.x >> 5;
    for (uint32_t r = ty; r < 32; r += 8) {
        const uint32_t k = k0 + r, b = b0 + tx;
        float v = 0.0f;
        if (k < p.K && b < blocks_per_row) {
            const size_t blk = (size_t)k * blocks_per_row + b;
            v = (p.absmax ? __ldg(p.absmax + blk) : dq_scale(__ldg(p.scale_codes + blk), sos)) * w_down;
        }
        tile[r][tx] = v;
    }
    __syncthreads();
    for (uint32_t r = ty; r < 32; r += 8) {
        const uint32_t b = b0 + r, k = k0 + tx;
        if (k < p.K && b < blocks_per_row) p.scales_t[(size_t)b * p.K + k] = __float2half_rn(tile[tx][r]);
    }
}

// The adapter factor in the orientation and type the GEMM reads it in (the pre-pass reads the other one as it is).
// From B of type T:
//   bf16: b_t[n][j] = B[j][n]: exact.
//   f32:  b_t[n][j] = bf16(B[j][n]), b_t[n][r + j] = the bf16 of what that rounding left: as an adapter of rank 2 r
//         whose intermediate holds every column twice, B enters the product with sixteen bits of mantissa.
template <class T>
__device__ __forceinline__ void repack_adapter_block(const RepackParams &p, uint32_t block, float (*tile)[33]) {
    constexpr bool kF32 = sizeof(T) == 4;
    // a tile of 32 x 32 of the result [N][r]
    const T *src = static_cast<const T *>(p.b);
    const uint32_t rows = p.N, cols = p.r, col_tiles = (cols + 31) / 32;
    const uint32_t r0 = block / col_tiles * 32, c0 = block % col_tiles * 32, tx = threadIdx.x & 31u, ty = threadIdx.x >> 5;
    #pragma unroll
    for (uint32_t q = ty; q < 32; q += 8) {
        const uint32_t r = r0 + (p.factor_out_in ? q : tx), c = c0 + (p.factor_out_in ? tx : q);
        float v = 0.0f;
        if (r < rows && c < cols) v = (float)src[p.factor_out_in ? (size_t)r * cols + c : (size_t)c * rows + r];
        tile[r - r0][c - c0] = v;
    }
    __syncthreads();
    #pragma unroll
    for (uint32_t q = ty; q < 32; q += 8) {
        const uint32_t r = r0 + q, c = c0 + tx;
        if (r >= rows || c >= cols) continue;
        const float v = tile[q][tx];
        const __nv_bfloat16 hi = __float2bfloat16_rn(v);
        p.b_t[(size_t)r * (kF32 ? 2 * cols : cols) + c] = hi;
        if (kF32) p.b_t[(size_t)r * 2 * cols + cols + c] = __float2bfloat16_rn(v - __bfloat162float(hi));
    }
}

// The first code_blocks CTAs take the nibbles, the next scale_blocks the scales, the last adapter_blocks the adapter.  The
// launch runs beside the pre-pass ahead of it, which it shares nothing with (and which lets it start once the kernels
// before have completed): one CTA waits for that at the end, so that whoever waits for this kernel finds both complete.
// (Weight first, pre-pass beside it: the pre-pass's CTAs found no room until the many small ones were through.  Both in one
// launch, whose CTAs have the pre-pass's registers: 512 x 4096 x 4096 in f32 0.3 to 1.3 us longer.)
template <class T>
__global__ void __launch_bounds__(256) repack_kernel(const RepackParams p) {
    __shared__ __align__(16) uint32_t smem[128 * 32];
    ptx::pdl_launch_dependents();
    const uint32_t b = blockIdx.x;
    if (b < p.code_blocks) repack_codes_block(p, b, smem);
    else if (b < p.code_blocks + p.scale_blocks) repack_scales_block(p, b - p.code_blocks, reinterpret_cast<float(*)[33]>(smem));
    else repack_adapter_block<T>(p, b - p.code_blocks - p.scale_blocks, reinterpret_cast<float(*)[33]>(smem));
    if (b == 0) ptx::pdl_wait();
}

// ---- host side -----------------------------------------------------------------------
uint32_t lora_chunks_of(uint32_t rank) { return (rank + 63) / 64; }

}  // namespace

bool prefill_supported(const nf4_linear_args &a) {
    if (a.layout != NF4_LAYOUT_OUT_IN) return false;
    if (a.io_dtype != NF4_DTYPE_BF16 && a.io_dtype != NF4_DTYPE_F32) return false;
    const bool f32 = a.io_dtype == NF4_DTYPE_F32;
    if (a.rows <= 16) return false;  // the decode kernel's territory
    if (a.d_in % 64 != 0 || a.d_in >= (1ull << 31) || a.d_out >= (1ull << 31) || a.rows >= (1ull << 31))
        return false;
    const uint64_t ldy = a.ldy ? a.ldy : a.d_out;
    const uint64_t ybytes = (a.y_f32 || f32) ? 4 : 2;
    if ((ldy * ybytes) % 16 != 0 || !aligned16(a.y) || !aligned16(a.x) || !aligned16(a.packed))
        return false;
    if (a.lora_a && f32) {
        // f32 factors are converted into the workspace and enter as an adapter of twice the rank
        if (2 * a.lora_rank > 256 || (2 * a.lora_rank) % 8 != 0) return false;
    } else if (a.lora_a) {
        // LoRA B is read by TMA: rows (rank * 2 bytes) must be a multiple of 16 bytes
        if (a.lora_rank > 256 || a.lora_rank % 8 != 0 || !aligned16(a.lora_b)) return false;
        if (a.d_in % 8 != 0 || !aligned16(a.lora_a)) return false;
    }
    return true;
}

namespace {
// How the tiles are shared out between the pairs of CTAs: the first `sk_tiles` tiles are divided by k-stages
// (every pair the same number of stages, a tile possibly split between neighbours), the other
// pairs * dp_rounds tiles go out whole.  With a tile count that is a multiple of the pairs nothing
// is split.  Otherwise the last round of whole tiles would leave most pairs idle, so the last full round and
// the remainder are divided by stages instead.  Fewer tiles than pairs: what of three takes the shortest (SharingCost): whole tiles;
// `split` pairs to a tile, whose sums a kernel of its own adds; or divided by stages, every pair 24 at least, with a tile's last pair
// collecting.
struct Sharing {
    uint32_t bn;  // activation rows of a tile
    uint32_t pairs, sk_tiles, dp_rounds, split;
    uint64_t cost;  // ns, if there are fewer tiles than pairs
};
// What a way to share fewer tiles than pairs takes, in ns, beside what all have in common: fitted to 3200 calls, back to back, of 450
// sizes from 17 x 256 x 256 to 1200 x 20480 x 20480 in both orientations and types, each in up to eight ways.  A stage is the dequantisers'
// time, or in a tile of many columns the MMAs'.  A read-out, or a dump, and the sums' launch grow with a tile's columns, the sums with
// all pairs' columns; and the more pairs, the fewer of their CTAs find an SM beside the pre-pass, to set themselves up in its shadow.
// Before, with 200 or 280 ns a stage whatever the columns and no word of the pairs -> now: 146 x 2176 x 1024 16.4 -> 15.4 us, 117 x 7680 x
// 704 24.2 -> 16.9, 62 x 1792 x 640 in the other orientation 16.3 -> 14.9, 1155 x 5888 x 2560 49.6 -> 43.2.  Of the 450 sizes 77 gain more
// than 2 %, 1.35 % on average; 15 lose more than 2 %, the most 10 % (22.2 -> 24.5 us).
struct SharingCost {
    uint64_t columns, stage;  // of a tile
    SharingCost(uint32_t bn, uint64_t rows) : columns(rows > bn ? bn : (rows + 31) / 32 * 32), stage(165) {
        if (bn > 128 && columns * 275 / 256 > stage) stage = columns * 275 / 256;
    }
    uint64_t work(uint64_t stages, uint64_t pairs) const { return stages * stage + pairs * 2100 / (kNumSMs / 2); }
    uint64_t read_out() const { return columns * 8400 / 256; }
    uint64_t whole(uint64_t ks, uint64_t tiles) const { return work(ks, tiles) + read_out(); }
    uint64_t split(uint64_t ks, uint64_t tiles, uint64_t s) const {
        return work((ks + s - 1) / s, tiles * s) + 2700 + columns * 5900 / 256 + tiles * s * columns * 2700 / (kNumSMs / 2 * 256);
    }
    uint64_t by_stages(uint64_t ks, uint64_t tiles, uint64_t pairs) const {
        return work(tiles * ks / pairs, pairs) + read_out() + 4000 + (pairs + tiles - 1) / tiles * 2200;
    }
};
Sharing share_tiles_of(uint32_t bn, uint64_t rows, uint64_t d_in, uint64_t d_out) {
    const uint64_t tiles = ((rows + bn - 1) / bn) * ((d_out + 2 * BM - 1) / (2 * BM)), ks = d_in / BK;
    Sharing sh{};
    sh.bn = bn;
    sh.split = 1;
    uint64_t pairs = kNumSMs / 2;
    if (tiles < pairs) {
        const SharingCost cost_of(bn, rows);
        const uint64_t by_stages = tiles * ks / 24, shared = by_stages < pairs ? by_stages : pairs;
        uint64_t least = cost_of.whole(ks, tiles), most = pairs / tiles;
        if (shared > tiles) {
            const uint64_t cost = cost_of.by_stages(ks, tiles, shared);
            if (cost < least) {
                least = cost;
                sh.split = 0;
            }
        }
        for (uint64_t s = 2; s <= most && s * 4 <= ks; ++s) {
            const uint64_t cost = cost_of.split(ks, tiles, s);
            if (cost < least) {
                least = cost;
                sh.split = (uint32_t)s;
            }
        }
        sh.cost = least;
        if (sh.split > 1) {
            sh.pairs = (uint32_t)(tiles * sh.split);
            sh.sk_tiles = (uint32_t)tiles;
            return sh;
        }
        pairs = sh.split ? tiles : shared;
        sh.split = 1;
    }
    sh.pairs = (uint32_t)pairs;
    if (tiles % pairs == 0) {
        sh.sk_tiles = 0;
        sh.dp_rounds = (uint32_t)(tiles / pairs);
    } else {
        sh.dp_rounds = tiles / pairs >= 1 ? (uint32_t)(tiles / pairs - 1) : 0u;
        sh.sk_tiles = (uint32_t)(tiles - (uint64_t)sh.dp_rounds * pairs);
    }
    return sh;
}
// Up to 128 rows there is one narrow tile where there would be a wide one.  More rows take narrow tiles where a pair gets one whole
// tile at most and that is the shorter way: 512 x 4096 x 4096 in 64 whole tiles instead of 32, two pairs to each and their sums added.
Sharing share_tiles(uint64_t rows, uint64_t d_in, uint64_t d_out, bool wide_only = false) {
    if (rows <= 128) return share_tiles_of(128, rows, d_in, d_out);
    const Sharing wide = share_tiles_of(256, rows, d_in, d_out);
    if (wide_only || !wide.cost) return wide;
    const uint64_t tiles = ((rows + 127) / 128) * ((d_out + 2 * BM - 1) / (2 * BM));
    if (tiles > kNumSMs / 2 || SharingCost(128, rows).whole(d_in / BK, tiles) >= wide.cost) return wide;
    Sharing sh{};
    sh.bn = 128;
    sh.split = sh.dp_rounds = 1;
    sh.pairs = (uint32_t)tiles;
    return sh;
}

struct WorkspaceLayout {
    uint64_t off_xh, off_scale, off_t, off_flags, off_partial, bytes;
    uint64_t off_b_t;                      // the adapter factor as the GEMM reads it (f32, other orientation)
    uint64_t off_codes_t, off_scales_t;    // the repacked weight (other orientation)
};
enum Extra { kPlain = 0, kFactor = 1, kFactorAndWeight = 2 };
// f16 copy of x | row scales | T (bf16 hi/lo) | flags and partial sums of the split tiles; d_in is
// bounded so that rows * d_in * 2 fits
WorkspaceLayout workspace_layout(uint64_t rows, uint64_t d_in, uint64_t d_out, uint32_t lora_rank,
                                 Extra extra = kPlain) {
    auto up = [](uint64_t v) { return (v + 255) / 256 * 256; };
    WorkspaceLayout w;
    w.off_xh = 256;  // the flag words at the start belong to the decode kernels and stay as they are
    w.off_scale = w.off_xh + up(rows * d_in * 2);
    w.off_t = w.off_scale + up(rows * 4);
    w.off_flags = w.off_t + up(rows * 2ull * 64 * lora_chunks_of(lora_rank) * 2);
    const Sharing sh = share_tiles(rows, d_in, d_out);
    w.off_partial = w.off_flags + up((uint64_t)sh.pairs * 8);
    w.bytes = w.off_partial + (sh.sk_tiles ? (uint64_t)sh.pairs * 2 * BM * sh.bn * 4 : 0);
    w.off_codes_t = w.off_scales_t = w.off_b_t = 0;
    if (extra >= kFactor) {  // `lora_rank` is the rank the GEMM sees (twice the adapter's for f32 factors)
        w.off_b_t = up(w.bytes);
        w.bytes = w.off_b_t + up(d_out * (uint64_t)lora_rank * 2);
    }
    if (extra >= kFactorAndWeight) {
        w.off_codes_t = up(w.bytes);
        w.off_scales_t = w.off_codes_t + up(d_in * d_out / 2);
        w.bytes = w.off_scales_t + up((d_out / 64) * d_in * 2);
    }
    return w;
}
}  // namespace

uint64_t prefill_workspace_bytes(uint64_t rows, uint64_t d_in, uint64_t d_out, uint32_t lora_rank) {
    if (rows <= 16 || d_in % 64 != 0 || d_in == 0 || d_out == 0) return 0;
    // f32 factors at worst; the other orientation where its shapes allow it
    return workspace_layout(rows, d_in, d_out, 2 * lora_rank, d_out % 64 == 0 ? kFactorAndWeight : kFactor).bytes;
}

// The reference's orientation (W [d_in][d_out], blocks along d_out) at more than 16 rows: repacked
// into the workspace, then the same GEMM.  Fewer rows stay with the CUDA-core strip kernel, whose
// f32 arithmetic is the reference's own.
bool prefill_in_out_supported(const nf4_linear_args &a) {
    if (a.layout != NF4_LAYOUT_IN_OUT) return false;
    if (a.io_dtype != NF4_DTYPE_BF16 && a.io_dtype != NF4_DTYPE_F32) return false;
    if (a.rows < kInOutMinRows) return false;
    if (a.d_in % 64 != 0 || a.d_out % 64 != 0 || a.d_in >= (1ull << 31) || a.d_out >= (1ull << 31) ||
        a.rows >= (1ull << 31))
        return false;
    const bool f32 = a.io_dtype == NF4_DTYPE_F32;
    const uint64_t ldy = a.ldy ? a.ldy : a.d_out;
    const uint64_t ybytes = (a.y_f32 || f32) ? 4 : 2;
    if ((ldy * ybytes) % 16 != 0 || !aligned16(a.y) || !aligned16(a.x) || !aligned16(a.packed)) return false;
    if (a.lora_a) {
        const uint32_t rank = f32 ? 2 * a.lora_rank : a.lora_rank;  // as the GEMM sees it
        if (rank > 256 || rank % 8 != 0) return false;
    }
    return true;
}

int32_t prefill_forward(const nf4_linear_args &a, cudaStream_t stream, void *r_out) {
    const bool repacked = a.layout == NF4_LAYOUT_IN_OUT;
    if (!(repacked ? prefill_in_out_supported(a) : prefill_supported(a)))
        return fail(NF4_ERR_UNSUPPORTED, "prefill_forward: unsupported shape");
    const bool x_f32 = a.io_dtype == NF4_DTYPE_F32;
    const bool y_f32 = a.y_f32 || x_f32;
    const Extra extra = repacked ? kFactorAndWeight : x_f32 ? kFactor : kPlain;
    PrefillParams p{};
    p.codes = a.packed;
    p.absmax = a.absmax;
    p.scale_codes = a.scale_codes;
    p.scale_of_scales = a.scale_of_scales;
    p.bias = a.bias;
    p.M = (uint32_t)a.rows;
    p.N = (uint32_t)a.d_out;
    p.K = (uint32_t)a.d_in;
    p.rank = a.lora_a ? a.lora_rank : 0;
    if (x_f32) p.rank *= 2;  // see repack_adapter_block
    p.lora_chunks = lora_chunks_of(p.rank);
    const Sharing sh = share_tiles(p.M, p.K, p.N);
    p.m_tiles = (p.M + sh.bn - 1) / sh.bn;
    // (the last tile's rows, if there is no other; of several tiles the last one's box is longer than it need be)
    p.box_rows = (p.m_tiles > 1 ? sh.bn : (p.M + 31) / 32 * 32) / 2;
    const uint64_t ldy = a.ldy ? a.ldy : a.d_out;
    if (p.N * (y_f32 ? 4u : 2u) % 16 != 0) p.y_ragged = a.y;
    p.ldy = ldy;

    const WorkspaceLayout wl = workspace_layout(p.M, p.K, p.N, p.rank, extra);
    if (a.workspace_bytes < wl.bytes) return fail(NF4_ERR_INVALID_ARG, "prefill_forward: workspace too small");
    p.sk_tiles = sh.sk_tiles;
    p.dp_rounds = sh.dp_rounds;
    p.split = sh.split;
    p.share_q = (uint64_t)sh.sk_tiles * (p.K / BK) / sh.pairs;
    p.share_r = (uint32_t)((uint64_t)sh.sk_tiles * (p.K / BK) % sh.pairs);
    p.wait_ns = 1000000000u;
    uint8_t *ws = static_cast<uint8_t *>(a.workspace);
    __half *xh = reinterpret_cast<__half *>(ws + wl.off_xh);
    float *row_scale = reinterpret_cast<float *>(ws + wl.off_scale);
    __nv_bfloat16 *t = reinterpret_cast<__nv_bfloat16 *>(ws + wl.off_t);
    p.row_scale = row_scale;
    p.sk_flags = reinterpret_cast<uint32_t *>(ws + wl.off_flags);
    p.partial = reinterpret_cast<float *>(ws + wl.off_partial);
    const void *lora_b = a.lora_b;
    RepackParams rp{};
    if (repacked) {  // the other orientation
        rp.codes = a.packed;
        rp.absmax = a.absmax;
        rp.scale_codes = a.scale_codes;
        rp.scale_of_scales = a.scale_of_scales;
        rp.codes_t = ws + wl.off_codes_t;
        rp.scales_t = reinterpret_cast<__half *>(ws + wl.off_scales_t);
        rp.code_cols = (p.N + 127) / 128;
        rp.code_blocks = rp.code_cols * ((p.K + 255) / 256);
        rp.scale_cols = (p.N / 64 + 31) / 32;
        rp.scale_blocks = rp.scale_cols * ((p.K + 31) / 32);
        p.codes = rp.codes_t;
        p.scales_t = rp.scales_t;
    }
    if (p.rank && (repacked || x_f32)) {
        rp.b = a.lora_b;
        rp.r = a.lora_rank;
        rp.factor_out_in = !repacked;
        rp.b_t = reinterpret_cast<__nv_bfloat16 *>(ws + wl.off_b_t);
        rp.adapter_blocks = (a.lora_rank + 31) / 32 * ((p.N + 31) / 32);
        lora_b = rp.b_t;
    }
    rp.K = p.K;
    rp.N = p.N;
    PrepassArgs pre{};
    pre.x = a.x;
    pre.x_f32 = x_f32;
    pre.M = p.M;
    pre.K = p.K;
    pre.a = a.lora_a;
    pre.rank = a.lora_a ? a.lora_rank : 0;
    pre.k_major = repacked;
    pre.scale = a.lora_scale;
    pre.xh = xh;
    pre.row_scale = row_scale;
    pre.t_out = t;
    pre.r_out = r_out;
    pre.absmax = a.absmax;
    pre.scale_codes = a.scale_codes;
    pre.scale_of_scales = a.scale_of_scales;
    pre.flags = p.sk_flags;
    pre.n_flags = 2 * sh.pairs;
    NF4_TRY(activations_prepass(pre, stream));
    if (const uint32_t blocks = rp.code_blocks + rp.scale_blocks + rp.adapter_blocks) {
        count_launch();
        NF4_TRY(launch_maybe_overlapped(x_f32 ? repack_kernel<float> : repack_kernel<__nv_bfloat16>, dim3(blocks), dim3(256), 0, stream, true, rp));
    }

    CUtensorMap map_x, map_t, map_b, map_y, map_w, map_ahead, map_s;
    NF4_TRY(make_map(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.codes, p.N, p.K / 2, p.K / 2, BM, BK, CU_TENSOR_MAP_SWIZZLE_64B));
    NF4_TRY(make_map(&map_ahead, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.codes, p.N, p.K / 2, p.K / 2, BM, 4 * BK, CU_TENSOR_MAP_SWIZZLE_NONE));
    const bool tma_scales = !repacked && (p.absmax ? p.K % 256 == 0 && aligned16(p.absmax) : p.K % 1024 == 0 && aligned16(p.scale_codes));
    map_s = map_w;
    if (repacked) NF4_TRY(make_map(&map_s, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, p.scales_t, p.N / 64, p.K, (uint64_t)p.K * 2, BM / 64, 2 * BK, CU_TENSOR_MAP_SWIZZLE_NONE));
    if (tma_scales && p.absmax)
        NF4_TRY(make_map(&map_s, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, p.absmax, p.N, p.K / 64, p.K / 16, BM, 4, CU_TENSOR_MAP_SWIZZLE_NONE));
    else if (tma_scales)
        NF4_TRY(make_map(&map_s, CU_TENSOR_MAP_DATA_TYPE_UINT8, p.scale_codes, p.N, p.K / 64, p.K / 64, BM, 16, CU_TENSOR_MAP_SWIZZLE_NONE));
    NF4_TRY(make_map(&map_x, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, xh, p.M, p.K, (uint64_t)p.K * 2, p.box_rows, BK,
                     CU_TENSOR_MAP_SWIZZLE_128B));
    map_t = map_b = map_x;
    if (p.rank) {
        const uint32_t ld_t = 2 * 64 * p.lora_chunks;
        NF4_TRY(make_map(&map_t, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, t, p.M, ld_t, (uint64_t)ld_t * 2, p.box_rows,
                         BK, CU_TENSOR_MAP_SWIZZLE_128B));
        // LoRA B [N][rank]: columns beyond the rank and rows beyond N read as zero
        NF4_TRY(make_map(&map_b, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, lora_b, p.N, p.rank,
                         (uint64_t)p.rank * 2, BM, BK, CU_TENSOR_MAP_SWIZZLE_128B));
    }
    if (y_f32)
        NF4_TRY(make_map(&map_y, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, a.y, p.M, p.N, ldy * 4, kEpiBytes / (BM * 4), BM,
                         CU_TENSOR_MAP_SWIZZLE_NONE));
    else
        NF4_TRY(make_map(&map_y, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, a.y, p.M, p.N, ldy * 2, kEpiBytes / (BM * 2), BM / 2,
                         CU_TENSOR_MAP_SWIZZLE_128B));

    auto go = [&](auto kernel) -> int32_t {
        NF4_TRY(ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), (int)kDynamicSmem));
        return launch_maybe_overlapped(kernel, dim3(2 * sh.pairs), dim3(kThreads), kDynamicSmem, stream, true, map_x, map_t, map_b,
                                       map_y, map_w, map_ahead, map_s, p);
    };
    auto pick = [&](auto bn) -> int32_t {
        constexpr int BN = decltype(bn)::value;
        if (repacked) return y_f32 ? go(prefill_kernel<BN, true, kScalesPerK>) : go(prefill_kernel<BN, false, kScalesPerK>);
        if (tma_scales) return y_f32 ? go(prefill_kernel<BN, true, kScalesTma>) : go(prefill_kernel<BN, false, kScalesTma>);
        return y_f32 ? go(prefill_kernel<BN, true, kScalesLoaded>) : go(prefill_kernel<BN, false, kScalesLoaded>);
    };
    using Wide = std::integral_constant<int, 256>;
    using Narrow = std::integral_constant<int, 128>;
    NF4_TRY(sh.bn == 128 ? pick(Narrow{}) : pick(Wide{}));
    count_launch();
    NF4_TRY(check_cuda(cudaGetLastError(), "prefill_kernel launch"));
    if (sh.split <= 1) return NF4_OK;
    const uint32_t columns = p.M < sh.bn ? p.M : sh.bn;
    count_launch();
    auto sum = sh.bn == 128 ? (y_f32 ? sum_parts_kernel<128, true> : sum_parts_kernel<128, false>)
                            : (y_f32 ? sum_parts_kernel<256, true> : sum_parts_kernel<256, false>);
    return launch_maybe_overlapped(sum, dim3((columns + 7) / 8, sh.pairs / sh.split * 2), dim3(256), 0,
                                   stream, true, p.partial, p.split, p.m_tiles, p.M, p.N, p.row_scale, p.bias, a.y, ldy);
}


int32_t prefill_set_host_flag(int *mapped) {
    return check_cuda(cudaMemcpyToSymbol(g_prefill_error_host, &mapped, sizeof(mapped)), "setting the mapped failure word");
}

int32_t prefill_code_place(uint32_t block, uint32_t *slot_full_parity) {
    const CodePlace c = code_place(block);
    slot_full_parity[0] = c.slot;
    slot_full_parity[1] = c.full;
    slot_full_parity[2] = c.parity;
    return kCodeSlots;
}

// The sharing of the tiles, for inspection on the host, in tiles of 128 weight rows x *tile_rows activation rows, one CTA's part of a
// pair's tile: as a forward has it, or (wide_only) as it would be with 256 rows to a tile wherever there are more than 128.  CTAs are
// counted with the even ones of all pairs first: CTA `cta` is CTA cta / pairs of pair cta % pairs.  Returns the number of the CTA's
// segments (at most `cap` are written), or -1.
int32_t prefill_share_plan(uint64_t rows, uint64_t d_in, uint64_t d_out, bool wide_only, uint32_t cta, uint32_t *tile_rows, uint32_t *ctas,
                           uint32_t *segments, uint32_t cap) {
    if (rows <= 16 || d_in % BK != 0 || d_in == 0 || d_out == 0) return -1;
    const Sharing sh = share_tiles(rows, d_in, d_out, wide_only);
    if (tile_rows) *tile_rows = sh.bn;
    if (ctas) *ctas = 2 * sh.pairs;
    if (cta >= 2 * sh.pairs) return -1;
    const uint32_t rank = cta / sh.pairs, m_tiles = (uint32_t)((rows + sh.bn - 1) / sh.bn);
    PrefillParams p{};
    p.sk_tiles = sh.sk_tiles;
    p.dp_rounds = sh.dp_rounds;
    p.split = sh.split;
    p.share_q = (uint64_t)sh.sk_tiles * (d_in / BK) / sh.pairs;
    p.share_r = (uint32_t)((uint64_t)sh.sk_tiles * (d_in / BK) % sh.pairs);
    WorkList wl;
    wl.init(p, (uint32_t)(d_in / BK), cta % sh.pairs, sh.pairs);
    uint32_t n = 0;
    for (uint32_t j = 0; j < wl.n_seg; ++j) {
        uint32_t tile, b, e;
        wl.get(j, tile, b, e);
        const uint32_t n_tile = tile / m_tiles * 2 + rank;
        if ((uint64_t)n_tile * BM >= d_out) continue;  // the odd CTA of the last pair of an odd number of tiles: no rows
        if (n < cap) {
            segments[3 * n] = n_tile * m_tiles + tile % m_tiles;
            segments[3 * n + 1] = b;
            segments[3 * n + 2] = e;
        }
        ++n;
    }
    return (int32_t)n;
}

int32_t prefill_error_flag_ptr(int **dev_ptr) {
    return check_cuda(cudaGetSymbolAddress(reinterpret_cast<void **>(dev_ptr), g_prefill_error),
                      "address of the prefill error flag");
}

int32_t prefill_failure_ref(FailureRef *ref) {
    static std::mutex mu;
    static FailureRef of_device[64] = {};
    int dev = 0;
    NF4_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(NF4_ERR_UNSUPPORTED, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(mu);
    if (!of_device[dev].flag) {
        void *host = nullptr;
        int *flag = nullptr;
        NF4_CUDA_TRY(cudaGetSymbolAddress(&host, g_prefill_error_host));
        NF4_TRY(prefill_error_flag_ptr(&flag));
        of_device[dev] = FailureRef{flag, static_cast<int **>(host)};
    }
    *ref = of_device[dev];
    return NF4_OK;
}

}  // namespace nf4
