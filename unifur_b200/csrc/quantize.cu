// Blockwise-absmax NF4 quantize / dequantize / double-quantize kernels (sm_100a).
//
// All four are HBM-bound streaming kernels: 4.5625 algorithmic bytes per value
// (4 B of f32 on one side, 0.5 B of nibbles + 4/64 B of absmax on the other).
// Layout: values and outputs are flat arrays; a thread owns 8 consecutive values
// (one 32-byte sector of f32, one 32-bit word of nibbles), 8 lanes own one
// 64-value block, a warp owns 4 blocks, and warps stride over the array.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "kernels.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace nf4 {

namespace {

constexpr int kThreads = 256;
constexpr int kWarpsPerCta = kThreads / 32;

// End of a kernel that writes weights.  The forward kernels ask for weights before they wait for the
// kernel ahead of them (programmatic launches), so these kernels let their successor start no sooner
// than their CTAs end, with what they wrote visible by then.
__device__ __forceinline__ void publish_weight() { __threadfence(); }

// Copies the cell table of the fast code selection into shared memory (a barrier must follow).
__device__ __forceinline__ void load_cells(uint32_t *cells) {
    if (threadIdx.x < kCellWords) cells[threadIdx.x] = c_cell_table[threadIdx.x];
}

__device__ __forceinline__ float group8_max(float m) {
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 1));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 2));
    m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, 4));
    return m;
}

// fold of |v| from 0.0 with maxNum: NaNs drop out exactly as f32::max does
__device__ __forceinline__ float absmax8(const float (&v)[8]) {
    float m = 0.0f;
    #pragma unroll
    for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(v[i]));
    return m;
}

// Eight consecutive f32: one load / store of a whole sector per thread where the buffer is 32-byte
// aligned (`wide`, the same for a whole launch), two of 16 bytes otherwise.
__device__ __forceinline__ void ld8_stream(const float *p, float (&v)[8], bool wide) {
    if (wide) {
        asm volatile("ld.global.cs.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7])
                     : "l"(p));
    } else {
        const float4 a = __ldcs(reinterpret_cast<const float4 *>(p)), b = __ldcs(reinterpret_cast<const float4 *>(p) + 1);
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    }
}
__device__ __forceinline__ void st8_stream(float *p, const float (&v)[8], bool wide) {
    if (wide) {
        asm volatile("st.global.cs.v8.f32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]),
                     "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "l"(p)
                     : "memory");
    } else {
        __stcs(reinterpret_cast<float4 *>(p), make_float4(v[0], v[1], v[2], v[3]));
        __stcs(reinterpret_cast<float4 *>(p) + 1, make_float4(v[4], v[5], v[6], v[7]));
    }
}

// One code per byte from eight nibbles.
__device__ __forceinline__ uint2 nibbles_to_bytes(uint32_t w) {
    const uint32_t even = w & 0x0f0f0f0fu, odd = (w >> 4) & 0x0f0f0f0fu;
    return make_uint2(__byte_perm(even, odd, 0x5140u), __byte_perm(even, odd, 0x7362u));
}

// One block of up to 64 values by a warp, two values per lane; a missing partner leaves its nibble 0.
template <bool PACKED>
__device__ __forceinline__ void quantize_block_by_warp(const float *values, uint32_t n, uint8_t *codes, float *absmax) {
    const uint32_t lane = threadIdx.x & 31u, e0 = 2 * lane;
    const bool h0 = e0 < n, h1 = e0 + 1 < n;
    const float x0 = h0 ? values[e0] : 0.0f;
    const float x1 = h1 ? values[e0 + 1] : 0.0f;
    float m = fmaxf(0.0f, fmaxf(fabsf(x0), fabsf(x1)));
    #pragma unroll
    for (int s = 1; s < 32; s <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    const uint32_t c0 = h0 ? code_of_exact(x0, m) : 0u;
    const uint32_t c1 = h1 ? code_of_exact(x1, m) : 0u;
    if (PACKED) {
        if (h0) codes[lane] = (uint8_t)(c0 | (c1 << 4));
    } else {
        if (h0) codes[e0] = (uint8_t)c0;
        if (h1) codes[e0 + 1] = (uint8_t)c1;
    }
    if (lane == 0) *absmax = m;
}

// 16-byte aligned buffers.  PACKED selects nibble packing (two codes per byte) versus one code per byte.
// `ngroups` groups of eight values make up the full 64-blocks; a ragged last block (`rest` values) is one
// more warp's work in the same launch.
// The loads of a warp's next chunk are in flight while it encodes one: without that a warp's 1 KB
// arrives, is encoded and only then replaced, and half of the time went to waiting (4096 x 4096 from
// rotating buffers: 15.4 us; 22.8 with the slower code selection and without that).
template <bool PACKED>
__global__ void __launch_bounds__(kThreads, 6)
quantize_full_kernel(const float *__restrict__ values, uint32_t ngroups, uint32_t rest,
                     uint8_t *__restrict__ codes, float *__restrict__ absmax, bool wide) {
    __shared__ uint32_t s_cells[kCellWords];
    load_cells(s_cells);
    __syncthreads();
    ptx::pdl_wait();
    // groups of eight values; eight neighbouring lanes hold a block, so a block's lanes are in range together
    const uint32_t step = gridDim.x * kThreads;
    uint32_t g = blockIdx.x * kThreads + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    float next[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (g < ngroups) ld8_stream(values + 8 * (uint64_t)g, next, wide);
    while (g - lane < ngroups) {
        float v[8];
        #pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = next[i];
        const uint32_t ahead = g + step;
        if (ahead < ngroups) ld8_stream(values + 8 * (uint64_t)ahead, next, wide);
        const float m = group8_max(absmax8(v));
        if (g < ngroups) {
            const uint32_t w = codes_of_group(v, m, s_cells);
            if (PACKED) reinterpret_cast<uint32_t *>(codes)[g] = w;
            else reinterpret_cast<uint2 *>(codes)[g] = nibbles_to_bytes(w);
            if ((lane & 7u) == 0) absmax[g >> 3] = m;
        }
        g = ahead;
    }
    if (rest && blockIdx.x == gridDim.x - 1 && threadIdx.x < 32)
        quantize_block_by_warp<PACKED>(values + 8 * (uint64_t)ngroups, rest, codes + (PACKED ? 4 : 8) * (uint64_t)ngroups,
                                       absmax + ngroups / 8);
    publish_weight();
}

// Buffers that are not 16-byte aligned: a warp per block.
template <bool PACKED>
__global__ void __launch_bounds__(kThreads)
quantize_generic_kernel(const float *__restrict__ values, uint64_t len, uint64_t nblocks, uint8_t *__restrict__ codes,
                        float *__restrict__ absmax) {
    const uint64_t warp = (uint64_t)blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5);
    const uint64_t nwarps = (uint64_t)gridDim.x * kWarpsPerCta;
    for (uint64_t blk = warp; blk < nblocks; blk += nwarps) {
        const uint64_t left = len - blk * kBlock;
        quantize_block_by_warp<PACKED>(values + blk * kBlock, left < kBlock ? (uint32_t)left : (uint32_t)kBlock,
                                       codes + blk * (PACKED ? kBlock / 2 : kBlock), absmax + blk);
    }
    publish_weight();
}

// ---- dequantize -------------------------------------------------------------

__device__ __forceinline__ float block_scale(const float *__restrict__ absmax,
                                             const uint8_t *__restrict__ scale_codes, float sos,
                                             uint64_t blk) {
    return absmax ? __ldg(absmax + blk) : dq_scale(__ldg(scale_codes + blk), sos);
}

// 16-byte aligned buffers.  A thread turns the codes of eight consecutive values into one 32-byte
// sector of output; four such groups are in flight per thread to cover the load latency.  The last
// len % 8 values go element by element.
template <bool PACKED>
__global__ void __launch_bounds__(kThreads, 8)
dequantize_full_kernel(const uint8_t *__restrict__ codes, uint32_t ngroups, uint32_t rest,
                       const float *__restrict__ absmax, const uint8_t *__restrict__ scale_codes,
                       const float *__restrict__ scale_of_scales, float *__restrict__ out, bool wide) {
    constexpr uint32_t kInFlight = 4;
    __shared__ float s_levels[16];
    if (threadIdx.x < 16) s_levels[threadIdx.x] = __uint_as_float(c_level_bits[threadIdx.x]);
    __syncthreads();
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();
    const float sos = scale_of_scales ? __ldg(scale_of_scales) : 0.0f;
    const uint32_t stride = gridDim.x * kThreads;
    for (uint32_t g0 = blockIdx.x * kThreads + threadIdx.x; g0 < ngroups; g0 += stride * kInFlight) {
        uint2 w[kInFlight];
        float s[kInFlight];
        #pragma unroll
        for (uint32_t u = 0; u < kInFlight; ++u) {
            const uint32_t g = g0 + u * stride;
            w[u] = make_uint2(0u, 0u);
            s[u] = 0.0f;
            if (g < ngroups) {
                if (PACKED) w[u].x = __ldcs(reinterpret_cast<const uint32_t *>(codes) + g);
                else w[u] = __ldcs(reinterpret_cast<const uint2 *>(codes) + g);
                s[u] = block_scale(absmax, scale_codes, sos, g >> 3);
            }
        }
        #pragma unroll
        for (uint32_t u = 0; u < kInFlight; ++u) {
            const uint32_t g = g0 + u * stride;
            if (g >= ngroups) continue;
            float v[8];
            #pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint32_t word = PACKED || i < 4 ? w[u].x : w[u].y;
                v[i] = __fmul_rn(s_levels[(word >> ((PACKED ? 4 * i : 8 * (i & 3)))) & 15u], s[u]);
            }
            st8_stream(out + 8 * (uint64_t)g, v, wide);
        }
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x < rest) {
        const uint64_t e = 8 * (uint64_t)ngroups + threadIdx.x;
        const uint32_t c = PACKED ? (uint32_t)codes[e >> 1] >> (4 * (e & 1u)) : codes[e];
        out[e] = __fmul_rn(s_levels[c & 15u], block_scale(absmax, scale_codes, sos, e / kBlock));
    }
}

template <bool PACKED>
__global__ void __launch_bounds__(kThreads)
dequantize_generic_kernel(const uint8_t *__restrict__ codes, uint64_t len,
                          const float *__restrict__ absmax,
                          const uint8_t *__restrict__ scale_codes,
                          const float *__restrict__ scale_of_scales, float *__restrict__ out) {
    const float sos = scale_of_scales ? __ldg(scale_of_scales) : 0.0f;
    const uint64_t stride = (uint64_t)gridDim.x * kThreads;
    for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < len; i += stride) {
        uint32_t c;
        if (PACKED) {
            const uint32_t byte = codes[i >> 1];
            c = (i & 1u) ? (byte >> 4) : (byte & 15u);
        } else {
            c = codes[i] & 15u;
        }
        const float s = block_scale(absmax, scale_codes, sos, i / kBlock);
        out[i] = __fmul_rn(__uint_as_float(c_level_bits[c]), s);
    }
}

// ---- load path: quantize the transpose of a checkpoint matrix without materialising it ----
// src is [rows, cols] row-major (a PyTorch linear weight [out, in], bf16 or f32); the result is
// the packed NF4 of its transpose [cols, rows] flattened row-major, i.e. element (c, r) at flat
// index c * rows + r.  With rows % 64 == 0 a 64-block of the result is 64 consecutive r for one
// c: a column segment of src.
// Two lanes (kSplit) share a column of f32, or a pair of columns of bf16 (one 32-bit word per row):
// each keeps 32 of the segment's 64 rows in registers, so a warp's load touches 64 bytes of two rows,
// 32 loads are in flight per thread, a block's maximum is one shuffle and its codes leave as one
// sector.  No shared-memory transpose.  CTAs that are neighbours in launch order take neighbouring row
// segments, so the sectors of an output line meet in the L2.
// Bound by instruction issue for a little over half of its time (14.7 per value, half of them to select
// the code: 23 us) and by waiting for its loads (28 warps an SM) and for the fence at the end.
// bf16 [14336, 4096]: 40 us; 92 through a 64 x 64 tile in shared memory with eight lanes per block; 49
// with all 64 rows in one thread's registers (twenty warps per SM) and with sixteen rows per thread
// (32-byte pieces of four rows per load: the L2 was busy with lookups).
constexpr int kTThreads = 128;
constexpr int kSplit = 2, kSplitRows = kBlock / kSplit, kSplitWords = 32 / kSplit;
constexpr int kTWords = kTThreads / kSplit;  // words (columns or pairs) a CTA covers

template <bool SRC_BF16>
__global__ void __launch_bounds__(kTThreads, 7)
quantize_transposed_kernel(const uint32_t *__restrict__ src, uint32_t segments, uint32_t words_per_row,
                           uint8_t *__restrict__ codes, float *__restrict__ absmax, bool wide) {
    __shared__ uint32_t s_cells[kCellWords];
    load_cells(s_cells);
    __syncthreads();
    ptx::pdl_wait();
    const uint32_t tile = blockIdx.x / segments, seg = blockIdx.x - tile * segments;
    const uint32_t lane = threadIdx.x & 31u, part = lane / kSplitWords;  // which 32 rows
    const uint32_t word = tile * kTWords + (threadIdx.x >> 5) * kSplitWords + lane % kSplitWords;
    const bool in = word < words_per_row;  // (the lanes of a word agree)
    const uint32_t *p = src + (uint64_t)(seg * kBlock + part * kSplitRows) * words_per_row + word;
    uint32_t w[kSplitRows];
    #pragma unroll
    for (int r = 0; r < kSplitRows; ++r, p += words_per_row) w[r] = in ? __ldcs(p) : 0u;
    uint32_t mx = 0;  // both columns' maxima of |bf16| as a pair (NaNs drop out), or the f32 column's
    auto larger = [&](uint32_t v) {
        if (SRC_BF16) asm("max.bf16x2 %0, %0, %1;" : "+r"(mx) : "r"(v & 0x7fff7fffu));
        else mx = __float_as_uint(fmaxf(__uint_as_float(mx), fabsf(__uint_as_float(v))));
    };
    #pragma unroll
    for (int r = 0; r < kSplitRows; ++r) larger(w[r]);
    #pragma unroll
    for (int s = kSplitWords; s < 32; s <<= 1) larger(__shfl_xor_sync(0xffffffffu, mx, s));
    if (!in) return;
    constexpr int kCols = SRC_BF16 ? 2 : 1;
    #pragma unroll 1  // (unrolled, both columns' values would be kept in registers at once)
    for (int h = 0; h < kCols; ++h) {
        const uint32_t half = h == 0 ? 0x1044u : 0x3244u;
        auto value = [&](uint32_t bits) { return __uint_as_float(SRC_BF16 ? __byte_perm(bits, 0u, half) : bits); };
        const float m = value(mx);
        const uint64_t blk = (uint64_t)(word * kCols + h) * segments + seg;  // the block's number in the result
        uint32_t out[kSplitRows / 8];
        #pragma unroll
        for (int g = 0; g < kSplitRows / 8; ++g) {
            float v[8];
            #pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = value(w[8 * g + i]);
            out[g] = codes_of_group(v, m, s_cells);
        }
        uint32_t *dst = reinterpret_cast<uint32_t *>(codes + blk * (kBlock / 2) + part * (kSplitRows / 2));
        if (wide) {
            *reinterpret_cast<uint4 *>(dst) = make_uint4(out[0], out[1], out[2], out[3]);
        } else {  // codes only 4-byte aligned
            #pragma unroll
            for (int g = 0; g < kSplitRows / 8; ++g) dst[g] = out[g];
        }
        if (part == 0) absmax[blk] = m;
    }
    publish_weight();
}
static_assert(kSplitRows == 32, "a lane stores four words of codes per block");

// The same where TMA takes the matrix (rows of whole 16-byte pieces): a warp takes a 64-block's rows of 32 words (64 columns of
// bf16, 32 of f32), a lane the 64 rows of a word.  The 8 KB come by TMA into the warp's own place in shared memory, pass into
// registers, and the next ones are asked for before these are encoded: the loads of sixteen warps, 128 KB an SM, are in flight
// while the codes of 128 values a lane are computed, where the kernel above loads, waits and computes in turn.  bf16 needs no
// look at the threshold's neighbourhood (see codes_of_bf16): 9 instructions a value.
constexpr int kTmaWarps = 8, kTmaThreads = kTmaWarps * 32, kTmaTile = kBlock * 128;  // two CTAs on an SM
constexpr uint32_t kTmaSmem = kTmaWarps * kTmaTile + 1024;

template <bool SRC_BF16>
__global__ void __launch_bounds__(kTmaThreads, 2)
quantize_transposed_tma_kernel(const __grid_constant__ CUtensorMap tmap, uint32_t segments, uint32_t octets, uint32_t words_per_row, uint32_t tiles,
                               uint8_t *__restrict__ codes, float *__restrict__ absmax, bool wide, uint32_t scales_at_once,
                               float *__restrict__ maxima, const FailureRef failure) {
    extern __shared__ uint8_t smem_any[];
    __shared__ uint32_t s_cells[kCellWords];
    __shared__ __align__(8) uint64_t s_bars[kTmaWarps];
    constexpr int kCols = SRC_BF16 ? 2 : 1;  // of a word
    __shared__ float s_max[2][kTmaWarps][32 * kCols];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    uint8_t *const place = smem_any + (1024u - (ptx::smem_addr(smem_any) & 1023u)) % 1024u + warp * kTmaTile;
    const uint32_t bar = ptx::smem_addr(s_bars + warp), stride = gridDim.x;
    if (threadIdx.x < kCellWords) s_cells[threadIdx.x] = SRC_BF16 ? c_cell_bf16_table[threadIdx.x] : c_cell_table[threadIdx.x];
    if (lane == 0) {
        ptx::mbar_init(bar, 1);
        ptx::fence_mbar_init();
        ptx::fence_proxy_async();
        if (warp == 0) ptx::prefetch_tmap(&tmap);
    }
    __syncthreads();
    ptx::pdl_wait();
    // A tile of the CTA: 32 words of eight segments, one a warp, so that a column's block scales are a sector and its codes two
    // lines.  The segments run fastest over the grid.
    auto request = [&](uint32_t tile) {
        const uint32_t group = tile / octets, seg = (tile - group * octets) * kTmaWarps + warp;
        if (seg >= segments) return;
        ptx::mbar_arrive_expect_tx(bar, kTmaTile);
        ptx::tma_load_2d(ptx::smem_addr(place), &tmap, (int32_t)(group * 32), (int32_t)(seg * kBlock), bar);
    };
    uint32_t parity = 0, turn = 0;
    float most = 0.0f;  // the largest scale so far, of the lane's columns
    bool lost = false;
    if (lane == 0 && blockIdx.x < tiles) request(blockIdx.x);
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += stride, turn ^= 1u) {
        const uint32_t group = tile / octets, seg0 = (tile - group * octets) * kTmaWarps, seg = seg0 + warp, word = group * 32 + lane;
        const bool mine = seg < segments && !lost;  // (the last tile of a group may have fewer segments)
        if (mine && !ptx::mbar_wait_suspended(bar, parity)) {
            lost = true;  // its codes are void, and no more tiles are asked for
            if (lane == 0) NF4_REPORT_FAILURE(*failure.flag, *failure.host, 15);
            ptx::let_flights_land();
        }
        if (mine) parity ^= 1u;
        uint32_t w[kBlock];
        #pragma unroll
        for (int r = 0; r < kBlock; ++r) w[r] = *reinterpret_cast<const uint32_t *>(place + r * 128 + lane * 4);
        uint32_t mx = 0;  // both columns' maxima of |bf16| as a pair (a NaN stays one), or the f32 column's (NaNs drop out)
        #pragma unroll
        for (int r = 0; r < kBlock; ++r) {
            if (SRC_BF16) asm("max.NaN.xorsign.abs.bf16x2 %0, %0, %1;" : "+r"(mx) : "r"(w[r]));
            else mx = __float_as_uint(fmaxf(__uint_as_float(mx), fabsf(__uint_as_float(w[r]))));
        }
        __syncwarp();  // every value has been used: the place may be filled again
        if (lane == 0 && tile + stride < tiles && !lost) request(tile + stride);
        #pragma unroll 1  // (unrolled, both columns' values would be kept in registers at once)
        for (int h = mine && word < words_per_row ? 0 : kCols; h < kCols; ++h) {
            const uint32_t half = h == 0 ? 0x1044u : 0x3244u;
            auto value = [&](uint32_t bits) { return __uint_as_float(SRC_BF16 ? __byte_perm(bits, 0u, half) : bits); };
            float m = fabsf(value(mx));
            const uint64_t blk = (uint64_t)(word * kCols + h) * segments + seg;  // the block's number in the result
            uint32_t out[kBlock / 8];
            if (SRC_BF16 && m >= 1e-30f && m <= 1e30f) {
                const float rcp = approx_rcp(m), rcp_units = rcp * 2097152.0f, rcp_cells = rcp * 64.0f;
                #pragma unroll
                for (int g = 0; g < kBlock / 8; ++g) {
                    float v[8];
                    #pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = value(w[8 * g + i]);
                    out[g] = codes_of_bf16(v, rcp_units, rcp_cells, s_cells);
                }
            } else if (SRC_BF16) {  // NaNs among them, or a scale the reciprocal is not used for
                m = 0.0f;
                #pragma unroll
                for (int r = 0; r < kBlock; ++r) m = fmaxf(m, fabsf(value(w[r])));
                #pragma unroll
                for (int g = 0; g < kBlock / 8; ++g) {
                    out[g] = 0;
                    #pragma unroll
                    for (int i = 0; i < 8; ++i) out[g] |= code_of_exact(value(w[8 * g + i]), m) << (4 * i);
                }
            } else {
                #pragma unroll
                for (int g = 0; g < kBlock / 8; ++g) {
                    float v[8];
                    #pragma unroll
                    for (int i = 0; i < 8; ++i) v[i] = value(w[8 * g + i]);
                    out[g] = codes_of_group(v, m, s_cells);
                }
            }
            uint32_t *dst = reinterpret_cast<uint32_t *>(codes + blk * (kBlock / 2));
            if (wide) {
                asm volatile("st.global.v8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"r"(out[0]), "r"(out[1]), "r"(out[2]), "r"(out[3]),
                             "r"(out[4]), "r"(out[5]), "r"(out[6]), "r"(out[7]), "l"(dst) : "memory");
            } else {  // codes only 4-byte aligned
                #pragma unroll
                for (int g = 0; g < kBlock / 8; ++g) dst[g] = out[g];
            }
            s_max[turn][warp][lane * kCols + h] = m;
            most = fmaxf(most, m);
        }
        // The block scales of the tile: eight segments of a column by a thread, in one sector where they are whole.  (The next
        // tile's go to the other half, and nobody writes this one before all have passed the barrier of that tile.)
        __syncthreads();
        const uint32_t c = threadIdx.x, col = group * 32 * kCols + c;
        if (c < 32 * kCols && col < words_per_row * kCols) {
            float *dst = absmax + (uint64_t)col * segments + seg0;
            if (scales_at_once == 8) {
                asm volatile("st.global.v8.f32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"f"(s_max[turn][0][c]), "f"(s_max[turn][1][c]),
                             "f"(s_max[turn][2][c]), "f"(s_max[turn][3][c]), "f"(s_max[turn][4][c]), "f"(s_max[turn][5][c]),
                             "f"(s_max[turn][6][c]), "f"(s_max[turn][7][c]), "l"(dst) : "memory");
            } else if (scales_at_once == 4) {  // (their number is a multiple of four, the tile's as well)
                #pragma unroll
                for (uint32_t i = 0; i < kTmaWarps; i += 4)
                    if (seg0 + i < segments)
                        *reinterpret_cast<float4 *>(dst + i) = make_float4(s_max[turn][i][c], s_max[turn][i + 1][c], s_max[turn][i + 2][c], s_max[turn][i + 3][c]);
            } else {
                for (uint32_t i = 0; i < min((uint32_t)kTmaWarps, segments - seg0); ++i) dst[i] = s_max[turn][i][c];
            }
        }
    }
    if (maxima) {  // (scales are not negative, never NaN: their patterns order like integers)
        const uint32_t all = __reduce_max_sync(0xffffffffu, __float_as_uint(most));
        __syncthreads();  // (the last tile's scales have left)
        if (lane == 0) s_max[0][0][warp] = __uint_as_float(all);
        __syncthreads();
        if (threadIdx.x == 0) {
            #pragma unroll
            for (int w = 0; w < kTmaWarps; ++w) most = fmaxf(most, s_max[0][0][w]);
            maxima[blockIdx.x] = most;
        }
    }
    publish_weight();
}

// Any shape: the transpose written out as f32 (then quantized by the flat kernels).
template <bool SRC_BF16>
__global__ void __launch_bounds__(kThreads)
transpose_to_f32_kernel(const void *__restrict__ src, uint64_t rows, uint64_t cols,
                        float *__restrict__ out) {
    __shared__ float s_t[32][33];
    const uint64_t tiles_c = (cols + 31) / 32;
    const uint64_t r0 = (blockIdx.x / tiles_c) * 32, c0 = (blockIdx.x % tiles_c) * 32;
    const uint32_t tx = threadIdx.x & 31u, ty = threadIdx.x >> 5;  // 32 x 8
    for (uint32_t i = ty; i < 32; i += 8) {
        const uint64_t r = r0 + i, c = c0 + tx;
        float v = 0.0f;
        if (r < rows && c < cols)
            v = SRC_BF16 ? __bfloat162float(static_cast<const __nv_bfloat16 *>(src)[r * cols + c])
                         : static_cast<const float *>(src)[r * cols + c];
        s_t[i][tx] = v;
    }
    __syncthreads();
    for (uint32_t i = ty; i < 32; i += 8) {
        const uint64_t c = c0 + i, r = r0 + tx;
        if (r < rows && c < cols) out[c * rows + r] = s_t[tx][i];
    }
}

// ---- embedding: gather rows of a packed table and dequantize them ---------------------
// out[t][j] = level[code(ids[t] * d_model + j)] * scale(block of that element): the rows a batch
// of token ids selects, without materialising the table.  Blocks run over the flat table, so
// with d_model % 8 == 0 a group of eight consecutive elements of a row shares one 32-bit code
// word and one block scale; other widths take the element-wise path.  An id outside
// [0, n_embedding) yields a row of NaNs (the reference's gather would panic; a device kernel
// must not trap).
//
// A warp takes a segment of 1024 consecutive elements of a row, four groups of eight per lane with
// their loads in flight together; the row and segment come from one 32-bit division per warp (a
// 64-bit division per group and one group in flight took 13.8 us for 4096 rows of 3584 in bf16).
constexpr uint32_t kGatherGroups = 4;  // groups of eight per lane
template <bool BF16>
__global__ void __launch_bounds__(kThreads)
embedding_gather_kernel(const uint8_t *__restrict__ codes, const float *__restrict__ absmax,
                        const uint8_t *__restrict__ scale_codes,
                        const float *__restrict__ scale_of_scales, uint64_t n_embedding,
                        uint32_t groups_per_row, const int64_t *__restrict__ ids, uint32_t segments,
                        uint32_t work, void *__restrict__ out, bool wide) {
    __shared__ float s_levels[16];
    if (threadIdx.x < 16) s_levels[threadIdx.x] = __uint_as_float(c_level_bits[threadIdx.x]);
    __syncthreads();
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();
    const uint32_t item = blockIdx.x * kWarpsPerCta + (threadIdx.x >> 5), lane = threadIdx.x & 31u;
    if (item >= work) return;
    const uint32_t t = item / segments, g0 = (item - t * segments) * (32 * kGatherGroups) + lane;
    const int64_t id = __ldg(ids + t);
    const bool known = id >= 0 && (uint64_t)id < n_embedding;
    const float sos = scale_of_scales ? __ldg(scale_of_scales) : 0.0f;
    const uint64_t row = (uint64_t)(known ? id : 0) * groups_per_row;
    uint32_t w[kGatherGroups];
    float s[kGatherGroups];
    #pragma unroll
    for (uint32_t u = 0; u < kGatherGroups; ++u) {
        const uint32_t g = g0 + 32 * u;
        const bool in = known && g < groups_per_row;
        w[u] = in ? __ldg(reinterpret_cast<const uint32_t *>(codes) + row + g) : 0u;
        s[u] = in ? block_scale(absmax, scale_codes, sos, (row + g) >> 3) : __uint_as_float(0x7fc00000u);  // NaN
    }
    #pragma unroll
    for (uint32_t u = 0; u < kGatherGroups; ++u) {
        const uint32_t g = g0 + 32 * u;
        if (g >= groups_per_row) continue;
        float v[8];
        #pragma unroll
        for (int k = 0; k < 8; ++k) v[k] = __fmul_rn(s_levels[(w[u] >> (4 * k)) & 15u], s[u]);
        const uint64_t at = (uint64_t)t * groups_per_row + g;
        if (BF16) {
            uint32_t o[4];
            #pragma unroll
            for (int k = 0; k < 4; ++k) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
                o[k] = *reinterpret_cast<const uint32_t *>(&h);
            }
            reinterpret_cast<uint4 *>(out)[at] = make_uint4(o[0], o[1], o[2], o[3]);
        } else {
            st8_stream(static_cast<float *>(out) + 8 * at, v, wide);
        }
    }
}

// Widths that are no multiple of eight: element by element.
template <bool BF16>
__global__ void __launch_bounds__(kThreads)
embedding_gather_elements_kernel(const uint8_t *__restrict__ codes, const float *__restrict__ absmax,
                                 const uint8_t *__restrict__ scale_codes,
                                 const float *__restrict__ scale_of_scales, uint64_t n_embedding,
                                 uint64_t d_model, const int64_t *__restrict__ ids, uint64_t n_ids,
                                 void *__restrict__ out) {
    const float sos = scale_of_scales ? __ldg(scale_of_scales) : 0.0f;
    const uint64_t total = n_ids * d_model, stride = (uint64_t)gridDim.x * kThreads;
    for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < total; i += stride) {
        const uint64_t t = i / d_model, j = i - t * d_model;
        const int64_t id = __ldg(ids + t);
        float v = __uint_as_float(0x7fc00000u);
        if (id >= 0 && (uint64_t)id < n_embedding) {
            const uint64_t e = (uint64_t)id * d_model + j;
            const uint32_t byte = __ldg(codes + (e >> 1));
            const uint32_t c = (e & 1u) ? (byte >> 4) : (byte & 15u);
            v = __fmul_rn(__uint_as_float(c_level_bits[c]), block_scale(absmax, scale_codes, sos, e / kBlock));
        }
        if (BF16) reinterpret_cast<__nv_bfloat16 *>(out)[i] = __float2bfloat16_rn(v);
        else reinterpret_cast<float *>(out)[i] = v;
    }
}

// ---- double quantization ------------------------------------------------------
// c = round_half_away(s / max * 255) clamped to [0, 255]; 0 when max == 0 (src/quantize.rs:294-301).
// A NaN quotient (inf / inf) casts to 0 as Rust's `as u8`.

static __device__ __noinline__ uint32_t scale_code_exact(float s, float max_scale) {
    if (max_scale == 0.0f) return 0u;
    float q = roundf(__fmul_rn(__fdiv_rn(s, max_scale), 255.0f));
    q = fminf(fmaxf(q, 0.0f), 255.0f);  // NaN -> 0 through fmaxf
    return (uint32_t)q;
}

// The same without the division where that is safe: t = s * (255 / max) is within 1.2e-4 of the
// reference's product, so unless it lies within 2.5e-4 of a half (or is NaN, or the largest scale is
// outside the reciprocal's range) both round to the same integer.
struct ScaleEncoder {
    float max_scale, factor;
    bool ranged;
    __device__ explicit ScaleEncoder(float m)
        : max_scale(m), factor(255.0f * approx_rcp(m)), ranged(m >= 1e-30f && m <= 1e30f) {}
    __device__ __forceinline__ uint32_t four(const float4 &v) const {
        const float s[4] = {v.x, v.y, v.z, v.w};
        uint32_t c[4];
        bool sure = ranged;
        #pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float t = __fmul_rn(s[i], factor), r = t + 12582912.0f;  // t's nearest integer in the low mantissa bits
            sure = sure && fabsf(t - (r - 12582912.0f)) < 0.49975f;
            c[i] = __float_as_uint(r);
        }
        if (!sure) {
            #pragma unroll
            for (int i = 0; i < 4; ++i) c[i] = scale_code_exact(s[i], max_scale);
        }
        return __byte_perm(__byte_perm(c[0], c[1], 0x0040u), __byte_perm(c[2], c[3], 0x0040u), 0x5410u);
    }
};

// Pass 1 for up to kClusterMaxBlocks scales: the maximum by one cluster of sixteen CTAs, whose results
// meet in distributed shared memory, so that no word has to be cleared first.  Sixteen SMs with eight
// 16-byte loads in flight per thread read 3.7 MB (the scales of 14336 x 4096 weights) from the L2 in
// about 2 us.  (Both passes in one cluster: 16 us, the encoding is too much work for sixteen SMs.)
constexpr int kClusterCtas = 1 << (kClusterSizes - 1), kClusterThreads = 1024;
constexpr uint64_t kClusterMaxBlocks = 1u << 20;

__global__ void __launch_bounds__(kClusterThreads, 1)
scale_max_cluster_kernel(const float4 *__restrict__ absmax4, const float *__restrict__ absmax, uint32_t nblocks,
                         float *__restrict__ scale_of_scales) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ float s_warp[kClusterThreads / 32];
    __shared__ float s_cta[kClusterCtas];
    const uint32_t rank = cluster.block_rank(), tid = threadIdx.x;
    const uint32_t n4 = nblocks / 4;
    constexpr uint32_t kStride = kClusterCtas * kClusterThreads, kInFlight = 8;
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();
    cluster.barrier_arrive();  // (waited for before another CTA's shared memory is touched)
    float m = 0.0f;
    for (uint32_t i = rank * kClusterThreads + tid; i < n4; i += kStride * kInFlight) {
        float4 v[kInFlight];
        #pragma unroll
        for (uint32_t u = 0; u < kInFlight; ++u)
            v[u] = i + u * kStride < n4 ? __ldg(absmax4 + i + u * kStride) : make_float4(0.f, 0.f, 0.f, 0.f);
        #pragma unroll
        for (uint32_t u = 0; u < kInFlight; ++u) m = fmaxf(fmaxf(m, fmaxf(v[u].x, v[u].y)), fmaxf(v[u].z, v[u].w));
    }
    if (rank == 0 && 4 * n4 + tid < nblocks) m = fmaxf(m, __ldg(absmax + 4 * n4 + tid));
    #pragma unroll
    for (int s = 1; s < 32; s <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    if ((tid & 31u) == 0) s_warp[tid >> 5] = m;
    __syncthreads();
    if (tid < 32) {
        m = s_warp[tid];
        #pragma unroll
        for (int s = 1; s < 32; s <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    }
    cluster.barrier_wait();
    if (tid == 0) cluster.map_shared_rank(s_cta, 0)[rank] = m;
    cluster.sync();
    if (rank == 0 && tid == 0) {
        m = s_cta[0];
        #pragma unroll
        for (int r = 1; r < kClusterCtas; ++r) m = fmaxf(m, s_cta[r]);
        *scale_of_scales = m;
    }
}

// Both passes at once for up to kOneLaunchBlocks scales: the cluster's threads keep theirs (eight each) in registers
// while the maxima meet, every CTA gets all of them, and the codes follow without another launch and another reading.
// (The load of a bf16 [2048, 4096]: 13.8 -> 11.4 us; a round trip of 1.6 million values: 14.9 -> 13.7.  Beyond this size the
// encoding is too much for sixteen SMs.)
constexpr uint64_t kOneLaunchBlocks = (uint64_t)kClusterCtas * kClusterThreads * 8;

__global__ void __launch_bounds__(kClusterThreads, 1)
double_quantize_cluster_kernel(const float4 *__restrict__ absmax4, const float *__restrict__ absmax, uint32_t nblocks,
                               uint8_t *__restrict__ scale_codes, float *__restrict__ scale_of_scales, bool words) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ float s_warp[kClusterThreads / 32];
    __shared__ float s_cta[kClusterCtas];
    const uint32_t rank = cluster.block_rank(), tid = threadIdx.x, n4 = nblocks / 4, first = rank * kClusterThreads + tid;
    constexpr uint32_t kStride = kClusterCtas * kClusterThreads;
    cluster.barrier_arrive();  // (waited for before another CTA's shared memory is touched)
    ptx::pdl_wait();
    float4 v[2];
    #pragma unroll
    for (uint32_t u = 0; u < 2; ++u)
        v[u] = first + u * kStride < n4 ? __ldg(absmax4 + first + u * kStride) : make_float4(0.f, 0.f, 0.f, 0.f);
    const bool odd = rank == 0 && 4 * n4 + tid < nblocks;  // the last up to three
    const float last = odd ? __ldg(absmax + 4 * n4 + tid) : 0.0f;
    float m = last;
    #pragma unroll
    for (uint32_t u = 0; u < 2; ++u) m = fmaxf(fmaxf(m, fmaxf(v[u].x, v[u].y)), fmaxf(v[u].z, v[u].w));
    #pragma unroll
    for (int s = 1; s < 32; s <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    if ((tid & 31u) == 0) s_warp[tid >> 5] = m;
    __syncthreads();
    if (tid < 32) {
        m = s_warp[tid];
        #pragma unroll
        for (int s = 1; s < 32; s <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    }
    cluster.barrier_wait();
    if (tid < kClusterCtas) cluster.map_shared_rank(s_cta, tid)[rank] = m;
    cluster.sync();
    m = s_cta[0];
    #pragma unroll
    for (int r = 1; r < kClusterCtas; ++r) m = fmaxf(m, s_cta[r]);
    if (rank == 0 && tid == 0) *scale_of_scales = m;
    const ScaleEncoder enc(m);
    #pragma unroll
    for (uint32_t u = 0; u < 2; ++u) {
        const uint32_t i = first + u * kStride;
        if (i >= n4) continue;
        const uint32_t c = enc.four(v[u]);
        if (words) {
            reinterpret_cast<uint32_t *>(scale_codes)[i] = c;
        } else {
            #pragma unroll
            for (int b = 0; b < 4; ++b) scale_codes[4 * (size_t)i + b] = (uint8_t)(c >> (8 * b));
        }
    }
    if (odd) scale_codes[4 * (size_t)n4 + tid] = (uint8_t)scale_code_exact(last, m);
    publish_weight();
}

// More scales, unaligned ones, or a device that has no place for the cluster.  Pass 1: max over the (non-negative, never-NaN) block scales.  Their
// f32 bit patterns order like unsigned integers, so one atomicMax on the bits per warp is exact.
__global__ void __launch_bounds__(kThreads)
scale_max_kernel(const float *__restrict__ absmax, uint64_t nblocks, uint32_t *max_bits) {
    float m = 0.0f;
    const uint64_t stride = (uint64_t)gridDim.x * kThreads;
    #pragma unroll 4
    for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < nblocks; i += stride)
        m = fmaxf(m, __ldg(absmax + i));
    #pragma unroll
    for (int s = 1; s < 32; s <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, s));
    if ((threadIdx.x & 31u) == 0) atomicMax(max_bits, __float_as_uint(m));
}

// Pass 2, four scales per thread; `whole`: both buffers allow words of four.  The largest scale is the greatest of `n_maxima`
// values; where these are the quantizer's CTAs', this kernel is also the one that stores it.
__global__ void __launch_bounds__(kThreads)
scale_encode_kernel(const float *__restrict__ absmax, uint64_t nblocks, const float *maxima, uint32_t n_maxima, uint8_t *__restrict__ scale_codes,
                    float *scale_of_scales, bool whole) {
    __shared__ float s_warp[kWarpsPerCta];
    ptx::pdl_wait();
    const uint64_t stride = (uint64_t)gridDim.x * kThreads, first = (uint64_t)blockIdx.x * kThreads + threadIdx.x;
    const uint64_t n4 = whole ? nblocks / 4 : 0;
    float4 next = first < n4 ? __ldg(reinterpret_cast<const float4 *>(absmax) + first) : make_float4(0.f, 0.f, 0.f, 0.f);
    float max_scale = *maxima;
    if (n_maxima > 1) {
        for (uint32_t i = threadIdx.x; i < n_maxima; i += kThreads) max_scale = fmaxf(max_scale, maxima[i]);
        max_scale = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(max_scale)));
        if ((threadIdx.x & 31u) == 0) s_warp[threadIdx.x >> 5] = max_scale;
        __syncthreads();
        #pragma unroll
        for (int w = 0; w < kWarpsPerCta; ++w) max_scale = fmaxf(max_scale, s_warp[w]);
    }
    if (maxima != scale_of_scales && first == 0) *scale_of_scales = max_scale;
    const ScaleEncoder enc(max_scale);
    for (uint64_t i = first; i < n4; i += stride) {
        const float4 v = next;
        if (i + stride < n4) next = __ldg(reinterpret_cast<const float4 *>(absmax) + i + stride);
        reinterpret_cast<uint32_t *>(scale_codes)[i] = enc.four(v);
    }
    for (uint64_t i = 4 * n4 + first; i < nblocks; i += stride)
        scale_codes[i] = (uint8_t)scale_code_exact(__ldg(absmax + i), max_scale);
    publish_weight();
}

inline bool aligned32(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 31u) == 0; }

int grid_for(uint64_t work_items, int per_cta, int max_waves) {
    uint64_t ctas = (work_items + per_cta - 1) / per_cta;
    uint64_t cap = (uint64_t)kNumSMs * max_waves;
    if (ctas > cap) ctas = cap;
    if (ctas < 1) ctas = 1;
    return (int)ctas;
}

constexpr uint64_t kSliceBlocks = 1ull << 27;  // blocks one launch of a flat kernel takes

template <bool PACKED>
int32_t quantize_impl(const float *values, uint64_t len, uint8_t *codes, float *absmax,
                      cudaStream_t stream) {
    if (len == 0) return NF4_OK;
    if (!values || !codes || !absmax) return fail(NF4_ERR_INVALID_ARG, "nf4_quantize: null pointer");
    const uint64_t nblocks = (len + kBlock - 1) / kBlock;
    if (aligned16(values) && aligned16(codes) && ((uintptr_t)absmax % 4 == 0)) {
        for (uint64_t b0 = 0; b0 < nblocks; b0 += kSliceBlocks) {  // (32-bit positions in the kernel)
            const uint64_t left = len - b0 * kBlock, n = left < kSliceBlocks * kBlock ? left : kSliceBlocks * kBlock;
            count_launch();
            NF4_TRY(launch_maybe_overlapped(quantize_full_kernel<PACKED>, dim3(grid_for((n + 7) / 8, kThreads, 6)), dim3(kThreads), 0,
                                            stream, true, values + b0 * kBlock, (uint32_t)(n / kBlock * 8), (uint32_t)(n % kBlock),
                                            codes + b0 * (PACKED ? kBlock / 2 : kBlock), absmax + b0, aligned32(values)));
        }
        return NF4_OK;
    }
    quantize_generic_kernel<PACKED><<<grid_for(nblocks, kWarpsPerCta, 8), kThreads, 0, stream>>>(values, len, nblocks, codes, absmax);
    count_launch();
    return check_cuda(cudaGetLastError(), "nf4_quantize launch");
}

template <bool PACKED>
int32_t dequantize_impl(const uint8_t *codes, uint64_t len, const float *absmax,
                        const uint8_t *scale_codes, const float *scale_of_scales, float *out,
                        cudaStream_t stream) {
    if (len == 0) return NF4_OK;
    if (!codes || !out) return fail(NF4_ERR_INVALID_ARG, "nf4_dequantize: null pointer");
    if ((absmax != nullptr) == (scale_codes != nullptr))
        return fail(NF4_ERR_INVALID_ARG,
                    "nf4_dequantize: give either absmax or scale_codes+scale_of_scales");
    if (scale_codes && !scale_of_scales)
        return fail(NF4_ERR_INVALID_ARG, "nf4_dequantize: scale_codes without scale_of_scales");
    if (aligned16(codes) && aligned16(out)) {
        for (uint64_t b0 = 0; b0 * kBlock < len; b0 += kSliceBlocks) {  // (32-bit positions in the kernel)
            const uint64_t left = len - b0 * kBlock, n = left < kSliceBlocks * kBlock ? left : kSliceBlocks * kBlock;
            count_launch();
            NF4_TRY(launch_maybe_overlapped(dequantize_full_kernel<PACKED>, dim3(grid_for(n / 8, kThreads, 8)), dim3(kThreads), 0,
                                            stream, true, codes + b0 * (PACKED ? kBlock / 2 : kBlock), (uint32_t)(n / 8),
                                            (uint32_t)(n % 8), absmax ? absmax + b0 : nullptr, scale_codes ? scale_codes + b0 : nullptr,
                                            scale_of_scales, out + b0 * kBlock, aligned32(out)));
        }
        return NF4_OK;
    }
    dequantize_generic_kernel<PACKED><<<grid_for(len, kThreads, 8), kThreads, 0, stream>>>(codes, len, absmax, scale_codes,
                                                                                       scale_of_scales, out);
    count_launch();
    return check_cuda(cudaGetLastError(), "nf4_dequantize launch");
}

}  // namespace

int32_t quantize_packed(const float *values, uint64_t len, uint8_t *packed, float *absmax,
                        cudaStream_t stream) {
    return quantize_impl<true>(values, len, packed, absmax, stream);
}

int32_t quantize_unpacked(const float *values, uint64_t len, uint8_t *codes, float *absmax,
                          cudaStream_t stream) {
    return quantize_impl<false>(values, len, codes, absmax, stream);
}

int32_t dequantize_packed(const uint8_t *packed, uint64_t len, const float *absmax,
                          const uint8_t *scale_codes, const float *scale_of_scales, float *out,
                          cudaStream_t stream) {
    return dequantize_impl<true>(packed, len, absmax, scale_codes, scale_of_scales, out, stream);
}

int32_t dequantize_unpacked(const uint8_t *codes, uint64_t len, const float *absmax,
                            const uint8_t *scale_codes, const float *scale_of_scales, float *out,
                            cudaStream_t stream) {
    return dequantize_impl<false>(codes, len, absmax, scale_codes, scale_of_scales, out, stream);
}

int32_t quantize_transposed(const void *src, bool src_bf16, uint64_t rows, uint64_t cols,
                            uint8_t *packed, float *absmax, void *workspace, uint64_t workspace_bytes,
                            cudaStream_t stream, float *maxima, uint32_t *n_maxima) {
    if (n_maxima) *n_maxima = 0;
    if (rows == 0 || cols == 0) return NF4_OK;
    if (!src || !packed || !absmax) return fail(NF4_ERR_INVALID_ARG, "nf4_quantize_transposed: null pointer");
    const bool fused = rows % kBlock == 0 && cols % 4 == 0 && aligned16(src) &&
                       (reinterpret_cast<uintptr_t>(packed) & 3u) == 0;
    if (fused) {
        const uint64_t words = src_bf16 ? cols / 2 : cols;
        const uint64_t ctas = rows / kBlock * ((words + kTWords - 1) / kTWords);
        if (ctas >= (1ull << 31) || rows >= (1ull << 31) || cols >= (1ull << 31))
            return fail(NF4_ERR_UNSUPPORTED, "nf4_quantize_transposed: matrix too large");
        const uint32_t *w = static_cast<const uint32_t *>(src);
        count_launch();
        // The TMA kernel gains where its CTAs have enough to do for its later start and even shares of it; a tile is eight
        // segments of 32 words, those beyond the last segment included (back to back, cold, the other kernel's time first).
        // bf16: from 7/4 of the SMs in tiles on ([2048, 4096], 256 tiles: 9.7, 9.6 us; [4096, 4096] 15.9, 15.0; [14336, 7424]
        // 74, 57), and where most SMs have a tile and none two ([4096, 1024], 128: 7.2, 6.9; [3072, 1024], 96: 6.5, 6.6; [256, 4096]
        // 4.7, 5.3; [1536, 4096], 192: 8.4, 9.2), unless a fifth of the segments is missing ([1088, 11008], 17 of 24: 12.5, 13.4).
        // f32, bound by its bytes: 13/16 of the other kernel's time a segment and 2.6 us of start ([4096, 4096]: 19.5, 19.3;
        // [14336, 7424] 99, 84; [3584, 4096] 17.4, 17.5; [1024, 1024] 4.5, 6.3), more where the scales leave in less than sectors
        // ([4352, 7424], 68 segments: 31.8, 30.8; [4416, 4096], 69: 19.9, 20.7).
        const uint64_t segments = rows / kBlock, octets = (segments + kTmaWarps - 1) / kTmaWarps, strips = (words + 31) / 32, tiles = octets * strips;
        const bool even = tiles <= kNumSMs ? tiles * 4 >= kNumSMs * 3 : tiles * 4 >= kNumSMs * 7;
        const int64_t saved = (int64_t)strips * ((int64_t)segments * 16 - (int64_t)octets * kTmaWarps * 13);
        const bool gains = src_bf16 ? even && segments * 5 >= octets * kTmaWarps * 4 : saved >= (segments % 8 ? 35000 : 24576);
        if (words % 4 == 0 && gains) {
            auto kernel = src_bf16 ? quantize_transposed_tma_kernel<true> : quantize_transposed_tma_kernel<false>;
            CUtensorMap map;
            NF4_TRY(make_map(&map, CU_TENSOR_MAP_DATA_TYPE_UINT32, src, rows, words, words * 4, kBlock, 32, CU_TENSOR_MAP_SWIZZLE_NONE));
            FailureRef failure;
            NF4_TRY(prefill_failure_ref(&failure));
            NF4_TRY(ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), (int)kTmaSmem));
            const uint32_t ctas = (uint32_t)(tiles < 2 * kNumSMs ? tiles : 2 * kNumSMs);
            if (n_maxima) *n_maxima = ctas;
            return launch_maybe_overlapped(kernel, dim3(ctas), dim3(kTmaThreads), kTmaSmem, stream, true,
                                           map, (uint32_t)segments, (uint32_t)octets, (uint32_t)words, (uint32_t)tiles, packed, absmax, aligned32(packed),
                                           aligned32(absmax) && segments % 8 == 0 ? 8u : aligned16(absmax) && segments % 4 == 0 ? 4u : 1u, n_maxima ? maxima : nullptr, failure);
        }
        return launch_maybe_overlapped(src_bf16 ? quantize_transposed_kernel<true> : quantize_transposed_kernel<false>,
                                       dim3((unsigned)ctas), dim3(kTThreads), 0, stream, true, w, (uint32_t)(rows / kBlock), (uint32_t)words, packed, absmax,
                                       aligned16(packed));
    }
    // other shapes: transpose into the caller's workspace, then the flat quantizer
    const uint64_t need = rows * cols * sizeof(float);
    if (!workspace || workspace_bytes < need)
        return fail(NF4_ERR_INVALID_ARG,
                    "nf4_quantize_transposed: this shape needs a workspace of %llu bytes (rows %% 64 != 0)",
                    (unsigned long long)need);
    const uint64_t tiles = ((rows + 31) / 32) * ((cols + 31) / 32);
    if (tiles >= (1ull << 31)) return fail(NF4_ERR_UNSUPPORTED, "nf4_quantize_transposed: matrix too large");
    float *t = static_cast<float *>(workspace);
    if (src_bf16)
        transpose_to_f32_kernel<true><<<(unsigned)tiles, kThreads, 0, stream>>>(src, rows, cols, t);
    else
        transpose_to_f32_kernel<false><<<(unsigned)tiles, kThreads, 0, stream>>>(src, rows, cols, t);
    count_launch();
    NF4_CUDA_TRY(cudaGetLastError());
    return quantize_impl<true>(t, rows * cols, packed, absmax, stream);
}

int32_t embedding_gather(const uint8_t *packed, const float *absmax, const uint8_t *scale_codes,
                         const float *scale_of_scales, uint64_t n_embedding, uint64_t d_model,
                         const int64_t *ids, uint64_t n_ids, void *out, bool out_bf16,
                         cudaStream_t stream) {
    if (n_ids == 0 || d_model == 0) return NF4_OK;
    if (!packed || !ids || !out || (!absmax && !scale_codes))
        return fail(NF4_ERR_INVALID_ARG, "nf4_embedding_gather: null pointer");
    if (scale_codes && !scale_of_scales)
        return fail(NF4_ERR_INVALID_ARG, "nf4_embedding_gather: scale_codes without scale_of_scales");
    if ((d_model & 7u) == 0 && (!aligned16(out) || (reinterpret_cast<uintptr_t>(packed) & 3u)))
        return fail(NF4_ERR_INVALID_ARG, "nf4_embedding_gather: out must be 16-byte and packed 4-byte aligned");
    const uint64_t groups = d_model / 8, segments = (groups + 32 * kGatherGroups - 1) / (32 * kGatherGroups);
    if ((d_model & 7u) == 0 && groups < (1ull << 31) && n_ids * segments < (1ull << 31)) {
        const uint32_t work = (uint32_t)(n_ids * segments);
        const unsigned grid = (work + kWarpsPerCta - 1) / kWarpsPerCta;
        auto kernel = out_bf16 ? embedding_gather_kernel<true> : embedding_gather_kernel<false>;
        NF4_TRY(launch_maybe_overlapped(kernel, dim3(grid), dim3(kThreads), 0, stream, true, packed, absmax, scale_codes,
                                        scale_of_scales, n_embedding, (uint32_t)groups, ids, (uint32_t)segments, work, out,
                                        aligned32(out)));
    } else {
        auto kernel = out_bf16 ? embedding_gather_elements_kernel<true> : embedding_gather_elements_kernel<false>;
        kernel<<<grid_for(n_ids * d_model, kThreads, 16), kThreads, 0, stream>>>(packed, absmax, scale_codes, scale_of_scales,
                                                                                n_embedding, d_model, ids, n_ids, out);
    }
    count_launch();
    return check_cuda(cudaGetLastError(), "nf4_embedding_gather launch");
}

int32_t double_quantize(const float *absmax, uint64_t nblocks, uint8_t *scale_codes,
                        float *scale_of_scales, cudaStream_t stream) {
    if (!scale_of_scales) return fail(NF4_ERR_INVALID_ARG, "nf4_double_quantize: null scale_of_scales");
    if (nblocks == 0) return check_cuda(cudaMemsetAsync(scale_of_scales, 0, sizeof(float), stream), "nf4_double_quantize");
    if (!absmax || !scale_codes)
        return fail(NF4_ERR_INVALID_ARG, "nf4_double_quantize: null pointer");
    const bool whole = aligned16(absmax) && (reinterpret_cast<uintptr_t>(scale_codes) & 3u) == 0;
    const bool one_launch = aligned16(absmax) && nblocks <= kOneLaunchBlocks;
    ClusterRoom room;
    NF4_TRY(cluster_room(one_launch ? reinterpret_cast<const void *>(double_quantize_cluster_kernel)
                                    : reinterpret_cast<const void *>(scale_max_cluster_kernel), kClusterThreads, 0, &room));
    if (aligned16(absmax) && nblocks <= kClusterMaxBlocks && room.of[kClusterSizes - 1]) {
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(kClusterCtas);
        cfg.blockDim = dim3(kClusterThreads);
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = kClusterCtas;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        if (one_launch) {
            count_launch();
            return check_cuda(cudaLaunchKernelEx(&cfg, double_quantize_cluster_kernel, reinterpret_cast<const float4 *>(absmax), absmax,
                                                 (uint32_t)nblocks, scale_codes, scale_of_scales,
                                                 (reinterpret_cast<uintptr_t>(scale_codes) & 3u) == 0), "nf4_double_quantize launch");
        }
        NF4_TRY(check_cuda(cudaLaunchKernelEx(&cfg, scale_max_cluster_kernel, reinterpret_cast<const float4 *>(absmax), absmax,
                                              (uint32_t)nblocks, scale_of_scales), "nf4_double_quantize launch"));
    } else {
        NF4_CUDA_TRY(cudaMemsetAsync(scale_of_scales, 0, sizeof(float), stream));
        scale_max_kernel<<<grid_for(nblocks, kThreads * 4, 4), kThreads, 0, stream>>>(
            absmax, nblocks, reinterpret_cast<uint32_t *>(scale_of_scales));
        NF4_CUDA_TRY(cudaGetLastError());
    }
    count_launch(2);
    return launch_maybe_overlapped(scale_encode_kernel, dim3(grid_for(nblocks, kThreads * 4, 8)), dim3(kThreads), 0, stream, true,
                                   absmax, nblocks, static_cast<const float *>(scale_of_scales), 1u, scale_codes, scale_of_scales, whole);
}

uint64_t quantize_transposed_double_workspace_bytes(uint64_t rows, uint64_t cols) {
    const uint64_t plain = nf4_quantize_transposed_workspace_bytes(rows, cols), maxima = 2 * kNumSMs * sizeof(float);
    return plain > maxima ? plain : maxima;
}

// A kernel that reads all scales for their maximum, between the quantizer and the encoding, took 4 us of the 43 of a bf16
// [14336, 4096]; the quantizer's CTAs have it in passing.
int32_t quantize_transposed_double(const void *src, bool src_bf16, uint64_t rows, uint64_t cols, uint8_t *packed, float *absmax, uint8_t *scale_codes,
                                   float *scale_of_scales, void *workspace, uint64_t workspace_bytes, cudaStream_t stream) {
    if (!scale_of_scales || (rows && cols && !scale_codes)) return fail(NF4_ERR_INVALID_ARG, "nf4_quantize_transposed_double: null pointer");
    if (!workspace || workspace_bytes < quantize_transposed_double_workspace_bytes(rows, cols) || (reinterpret_cast<uintptr_t>(workspace) & 3u))
        return fail(NF4_ERR_INVALID_ARG, "nf4_quantize_transposed_double: workspace smaller than its bytes or not 4-byte aligned");
    float *maxima = static_cast<float *>(workspace);
    uint32_t n = 0;
    NF4_TRY(quantize_transposed(src, src_bf16, rows, cols, packed, absmax, workspace, workspace_bytes, stream, maxima, &n));
    const uint64_t nblocks = nf4_num_blocks(rows * cols);
    if (!n) return double_quantize(absmax, nblocks, scale_codes, scale_of_scales, stream);
    count_launch();
    return launch_maybe_overlapped(scale_encode_kernel, dim3(grid_for(nblocks, kThreads * 4, 8)), dim3(kThreads), 0, stream, true, absmax, nblocks,
                                   static_cast<const float *>(maxima), n, scale_codes, scale_of_scales,
                                   aligned16(absmax) && (reinterpret_cast<uintptr_t>(scale_codes) & 3u) == 0);
}

// ---- exhaustive self-check of the threshold bisection against the literal scan ----
// Walks `count` consecutive f32 bit patterns from `first_bits` and counts disagreements
// over the bisection's domain: NaNs and every value with |v| <= 65536.
__global__ void __launch_bounds__(kThreads)
selfcheck_codes_kernel(uint64_t first_bits, uint64_t count, unsigned long long *mismatches) {
    unsigned long long bad = 0;
    const uint64_t stride = (uint64_t)gridDim.x * kThreads;
    for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < count; i += stride) {
        const uint32_t bits = (uint32_t)(first_bits + i);
        const uint32_t mag = bits & 0x7fffffffu;
        if (mag > 0x47800000u && mag <= 0x7f800000u) continue;  // 65536 < |v| <= inf
        const float v = __uint_as_float(bits);
        bad += code_of_normalized(v) != code_by_scan(v);
    }
    if (bad) atomicAdd(mismatches, bad);
}

// Same walk for the division-free fast path: every f32 x with |x| <= absmax (and NaNs), one
// given absmax, compared with the exact division + literal scan.
__global__ void __launch_bounds__(kThreads)
selfcheck_fast_kernel(uint64_t first_bits, uint64_t count, float absmax,
                      unsigned long long *mismatches) {
    __shared__ uint32_t s_cells[kCellWords];
    load_cells(s_cells);
    __syncthreads();
    const bool rcp_ok = absmax >= 1e-30f && absmax <= 1e30f;
    const float rcp = approx_rcp(absmax);
    unsigned long long bad = 0;
    const uint64_t stride = (uint64_t)gridDim.x * kThreads;
    for (uint64_t i = (uint64_t)blockIdx.x * kThreads + threadIdx.x; i < count; i += stride) {
        const float x = __uint_as_float((uint32_t)(first_bits + i));
        if (fabsf(x) > absmax) continue;  // cannot occur inside a block whose absmax this is
        const uint32_t exact = absmax == 0.0f ? 7u : code_by_scan(__fdiv_rn(x, absmax));
        FastCodes f;
        f.take(x, rcp * 2097152.0f, rcp * 64.0f, s_cells);
        const uint32_t got = rcp_ok && f.sure() ? f.codes : code_of_exact(x, absmax);
        bad += got != exact;
    }
    if (bad) atomicAdd(mismatches, bad);
}

int32_t selfcheck_fast(uint64_t first_bits, uint64_t count, float absmax,
                       unsigned long long *mismatches_dev, cudaStream_t stream) {
    selfcheck_fast_kernel<<<kNumSMs * 8, kThreads, 0, stream>>>(first_bits, count, absmax,
                                                               mismatches_dev);
    count_launch();
    return check_cuda(cudaGetLastError(), "selfcheck launch");
}

int32_t selfcheck_codes(uint64_t first_bits, uint64_t count, unsigned long long *mismatches_dev,
                        cudaStream_t stream) {
    selfcheck_codes_kernel<<<kNumSMs * 8, kThreads, 0, stream>>>(first_bits, count, mismatches_dev);
    count_launch();
    return check_cuda(cudaGetLastError(), "selfcheck launch");
}

}  // namespace nf4
