// The reference's own orientation at few rows: y[M <= 16, N] = x W (+bias) (+ s (x A) B) with W [K, N],
// 64-blocks along N (src/qwennet.rs:230-241: linear(x, W[d_in, d_out])), d_out a multiple of 64, f32 or
// bf16 tensors, on CUDA cores in f32: every weight is its f32 level, the block's scale multiplies the
// activation of that k (one product for all the columns a lane has of the block), products and sums are
// f32.
//
// Split.  W is cut into strips of 256 columns; a strip's K into units of 64 rows; the units, strip by
// strip, are dealt out in equal contiguous runs, one per SM (11008 x 4096: 18.6 units each, 19 at most).
// A CTA works through its run segment by segment (a segment: the part of one strip it has).  Its warps take
// the rows of a segment in turn: a lane owns CPL consecutive columns, 256 / CPL lanes own a row, so a warp
// reads whole 128-byte lines of 32 CPL / 256 rows per step, D steps in flight in registers.
//
// Per weight.  One byte (two weights) indexes a 256-entry table of f32 pairs, replicated per lane (no bank
// conflicts).  The table lies at address 0x10000 of the shared window, so one byte permute of the code
// word with {8 lane, 0, 1, 0} is the whole address; the 64-bit entry is an operand of a packed
// multiply-add (fma.rn.f32x2) as it is.  Three instructions per two weights at one row (eight per weight
// in the kernel before, which scaled every weight, added the table's base and multiplied single f32).
// What bounds it.  At one row neither pipe: of 15.7 us (runs) the lookups' shared-memory wavefronts are 5.9 (two per lookup)
// and the instructions 4.4 (3.6 per weight with everything around the loop); the rest is latency at the ends of the
// segments: the first codes from idle, the barriers around a piece of x, the meeting of a strip's segments.  From
// about eight rows on the f32 rate.  f32 x [M, 4096], W [4096, 11008], f32
// scales, calls back to back, before -> now: 29.8 -> 16.4 us at one row, 36.4 -> 21.2 at four, 49.1 -> 31.2 at
// eight, 88.6 -> 55.9 at sixteen.
// Where there are few strips, a strip is a cluster's instead (template parameter CLUSTER): every CTA has one segment, and the
// strip's sums meet through distributed shared memory, in order, each CTA finishing a share of the columns (cluster_parts).
//
// Sums.  Lanes with the same columns meet by shuffles, the warps in shared memory, segments that share a
// strip in global memory, where the CTA that arrives last for a strip (a byte counter per strip in the
// workspace's flag words, zero at first use, left zero) adds them in the order of the runs: every sum has
// a fixed order.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "kernels.cuh"
#include "ptx.cuh"

namespace nf4 {
namespace {

constexpr uint32_t kStripCols = 256, kUnitRows = 64;
constexpr uint32_t kTableAt = 0x10000;                 // shared-window address of the table
constexpr uint32_t kRedBytes = 64 * 1024;              // behind the table: the warps' sums
constexpr uint32_t kXBytes = 60 * 1024;                // in front of it: activations of a piece of K
constexpr uint32_t kCounterStrips = 248;               // byte counters the flag words hold

struct StripParams {
    const void *x, *lora_b;
    void *y;
    const uint8_t *packed;
    const float *absmax;
    const uint8_t *scale_codes;
    const float *scale_of_scales;
    const float *bias;
    const float *t;        // [rows][rank] f32 = x A
    uint32_t *counters;
    float *partial;        // [2 per CTA][MR][256]
    uint32_t rows, K, N, rank;
    uint64_t ldy;
    float lora_scale;
    uint32_t units_per_strip, total_units;
    uint32_t whole_strips;  // runs are whole strips (more strips than counters)
    uint32_t parts;         // CLUSTER: a strip is a cluster's of so many CTAs, an equal part of its units each one's
    uint32_t x_rows;        // rows of W whose activations are in shared memory at a time
    uint32_t f32, y_f32, y_vec;
};

// floats between the activations of two rows of W in shared memory: padded so that the 16-byte stores of
// eight neighbouring rows fall into different banks
__host__ __device__ constexpr uint32_t x_stride(uint32_t mr) { return mr >= 8 ? mr + 4 : mr; }

__device__ __forceinline__ uint64_t dup(float v) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ void fma2(uint64_t &acc, uint64_t w, uint64_t x) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(w), "l"(x));
}
__device__ __forceinline__ void unpack(uint64_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

__host__ __device__ inline uint32_t run_begin(uint32_t total, uint32_t cta, uint32_t ctas) {
    return (uint32_t)((uint64_t)total * cta / ctas);
}
// the CTA whose run holds unit u
__device__ __forceinline__ uint32_t cta_of(uint32_t u, uint32_t total, uint32_t ctas) {
    uint32_t c = (uint32_t)(((uint64_t)u * ctas) / total);
    while (c + 1 < ctas && run_begin(total, c + 1, ctas) <= u) ++c;
    while (c > 0 && run_begin(total, c, ctas) > u) --c;
    return c;
}

// four neighbouring outputs of one row: adapter, bias, conversion, store
__device__ __forceinline__ void finish4(const StripParams &p, uint32_t m, uint32_t n, float4 v) {
    float o[4] = {v.x, v.y, v.z, v.w};
    if (p.rank) {
        float dot[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        #pragma unroll 4
        for (uint32_t j = 0; j < p.rank; ++j) {
            const float tv = __ldg(p.t + (size_t)m * p.rank + j);
            const size_t at = (size_t)j * p.N + n;
            #pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float bv = p.f32 ? __ldg(static_cast<const float *>(p.lora_b) + at + i)
                                       : __bfloat162float(static_cast<const __nv_bfloat16 *>(p.lora_b)[at + i]);
                dot[i] = fmaf(tv, bv, dot[i]);
            }
        }
        #pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = fmaf(dot[i], p.lora_scale, o[i]);
    }
    if (p.bias) {
        #pragma unroll
        for (int i = 0; i < 4; ++i) o[i] += __ldg(p.bias + n + i);
    }
    const size_t at = (size_t)m * p.ldy + n;
    if (p.f32 || p.y_f32) {
        float *y = static_cast<float *>(p.y) + at;
        if (p.y_vec) *reinterpret_cast<float4 *>(y) = make_float4(o[0], o[1], o[2], o[3]);
        else { y[0] = o[0]; y[1] = o[1]; y[2] = o[2]; y[3] = o[3]; }
    } else {
        __nv_bfloat16 *y = static_cast<__nv_bfloat16 *>(p.y) + at;
        const __nv_bfloat162 a = __floats2bfloat162_rn(o[0], o[1]), b = __floats2bfloat162_rn(o[2], o[3]);
        if (p.y_vec) *reinterpret_cast<uint2 *>(y) = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
        else { y[0] = a.x; y[1] = a.y; y[2] = b.x; y[3] = b.y; }
    }
}

template <int MR, int CPL, int THREADS, int D, bool DQ, bool CLUSTER>
__global__ void __launch_bounds__(THREADS, 1) in_out_strip_kernel(const StripParams p) {
    constexpr uint32_t kWarps = THREADS / 32, LPR = kStripCols / CPL, RS = 32 / LPR, kStep = kWarps * RS;
    constexpr int kWords = CPL / 8;
    constexpr uint32_t XS = x_stride(MR);
    constexpr int MG = (int)(kRedBytes / (kWarps * kStripCols * 4)) < MR ? (int)(kRedBytes / (kWarps * kStripCols * 4)) : MR;
    static_assert(kUnitRows % kStep == 0 && MR % MG == 0, "units are whole steps");
    extern __shared__ __align__(16) uint8_t dyn[];
    __shared__ uint32_t last_s;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t win = ptx::smem_addr(dyn), own = CLUSTER ? win & 0xff000000u : 0u;  // (a cluster's CTAs have their rank in the top byte)
    float *xs = reinterpret_cast<float *>(dyn);                             // [row of the piece][MR]
    uint8_t *table = dyn + ((own | kTableAt) - win);
    float *red = reinterpret_cast<float *>(table + 0x10000);                // [warp][MG][256]
    {
        // thread (byte, part) writes the copies of 32 * 256 / THREADS lanes, rotated over the banks
        constexpr uint32_t kParts = THREADS / 256, kCopies = 32 / kParts;
        const uint32_t byte = tid & 255u, part = tid >> 8;
        const float2 entry = make_float2(__uint_as_float(c_level_bits[byte & 15u]), __uint_as_float(c_level_bits[byte >> 4]));
        #pragma unroll 8
        for (uint32_t l = 0; l < kCopies; ++l)
            *reinterpret_cast<float2 *>(table + byte * 256u + ((part * kCopies + l + byte) & 31u) * 8u) = entry;
    }
    const float sos = DQ ? __ldg(p.scale_of_scales) : 0.0f;
    const uint32_t sub = lane / LPR, in_row = lane % LPR;
    const uint32_t lane_word = (lane * 8u) | kTableAt | own;  // bytes {8 lane, 0, 1, rank}
    const uint32_t blocks_per_row = p.N / kBlock;
    const uint32_t ctas = gridDim.x;
    uint32_t u = p.whole_strips ? run_begin(p.total_units / p.units_per_strip, blockIdx.x, ctas) * p.units_per_strip
                                : run_begin(p.total_units, blockIdx.x, ctas);
    const uint32_t run_end = p.whole_strips ? run_begin(p.total_units / p.units_per_strip, blockIdx.x + 1, ctas) * p.units_per_strip
                                          : run_begin(p.total_units, blockIdx.x + 1, ctas);
    const uint32_t cluster_strip = CLUSTER ? blockIdx.x / p.parts : 0u, cluster_part = CLUSTER ? blockIdx.x - cluster_strip * p.parts : 0u;
    const uint32_t u_end = CLUSTER ? cluster_strip * p.units_per_strip + run_begin(p.units_per_strip, cluster_part + 1, p.parts) : run_end;
    if (CLUSTER) u = cluster_strip * p.units_per_strip + run_begin(p.units_per_strip, cluster_part, p.parts);
    const uint32_t u_begin = u;
    bool first = true;
    while (u < u_end) {
        const uint32_t strip = u / p.units_per_strip, b = u - strip * p.units_per_strip;
        const uint32_t e = min(p.units_per_strip, b + (u_end - u));
        const uint32_t r0 = b * kUnitRows, r1 = min(e * kUnitRows, p.K);
        const uint32_t col = strip * kStripCols + in_row * CPL;
        const uint32_t row0 = r0 + warp * RS + sub;           // this lane's rows: row0, row0 + kStep, ...
        const uint8_t *code_at = p.packed + ((size_t)row0 * p.N + col) / 2;
        const size_t code_pitch = (size_t)kStep * p.N / 2;
        size_t scale_at = (size_t)row0 * blocks_per_row + col / kBlock;
        const size_t scale_pitch = (size_t)kStep * blocks_per_row;
        // rows this lane still has to ask for (none in columns beyond N)
        uint32_t to_fetch = col < p.N && row0 < r1 ? (r1 - row0 + kStep - 1) / kStep : 0u;

        uint32_t codes[D][kWords];
        uint32_t scale[D];
        auto fetch = [&](int d) {
            #pragma unroll
            for (int i = 0; i < kWords; ++i) codes[d][i] = 0;
            scale[d] = 0;
            if (to_fetch) {
                if constexpr (CPL == 32) {
                    const uint4 v = __ldcs(reinterpret_cast<const uint4 *>(code_at));
                    codes[d][0] = v.x; codes[d][1] = v.y; codes[d][2] = v.z; codes[d][3] = v.w;
                } else if constexpr (CPL == 16) {
                    const uint2 v = __ldcs(reinterpret_cast<const uint2 *>(code_at));
                    codes[d][0] = v.x; codes[d][1] = v.y;
                } else {
                    codes[d][0] = __ldcs(reinterpret_cast<const uint32_t *>(code_at));
                }
                scale[d] = DQ ? __ldg(p.scale_codes + scale_at) : __float_as_uint(__ldg(p.absmax + scale_at));
                --to_fetch;
            }
            code_at += code_pitch;
            scale_at += scale_pitch;
        };
        #pragma unroll
        for (int d = 0; d < D; ++d) fetch(d);
        if (first) {  // weights are immutable; x and T come from the kernels before this one
            ptx::pdl_wait();
            ptx::pdl_launch_dependents();
            first = false;
        }

        uint64_t acc[MR][CPL / 2];
        #pragma unroll
        for (int m = 0; m < MR; ++m)
            #pragma unroll
            for (int i = 0; i < CPL / 2; ++i) acc[m][i] = 0;
        for (uint32_t c0 = r0; c0 < r1; c0 += p.x_rows) {
            const uint32_t rows = min(p.x_rows, r1 - c0);  // of this piece of K; x_rows is a multiple of D * kStep
            const uint32_t steps = (rows + kStep - 1) / kStep;
            __syncthreads();  // (also: the table is in place)
            constexpr uint32_t kV = MR < 4 ? MR : 4;  // activation rows per store
            for (uint32_t i = tid; i < MR / kV * steps * kStep; i += THREADS) {
                const uint32_t mv = i / (steps * kStep), kk = i - mv * (steps * kStep);
                float v[kV];
                #pragma unroll
                for (uint32_t j = 0; j < kV; ++j) {
                    const uint32_t m = mv * kV + j;
                    const size_t at = (size_t)m * p.K + c0 + kk;
                    v[j] = 0.0f;
                    if (m < p.rows && kk < rows)
                        v[j] = p.f32 ? __ldg(static_cast<const float *>(p.x) + at)
                                     : __bfloat162float(static_cast<const __nv_bfloat16 *>(p.x)[at]);
                }
                float *dst = xs + kk * XS + mv * kV;
                if constexpr (kV == 4) *reinterpret_cast<float4 *>(dst) = make_float4(v[0], v[1], v[2], v[3]);
                else if constexpr (kV == 2) *reinterpret_cast<float2 *>(dst) = make_float2(v[0], v[1]);
                else *dst = v[0];
            }
            __syncthreads();
            const float *xrow = xs + (warp * RS + sub) * XS;
            auto multiply = [&](int d) {
                const float s = DQ ? dq_scale(scale[d], sos) : __uint_as_float(scale[d]);
                uint64_t xv[MR];
                if constexpr (MR >= 4) {
                    #pragma unroll
                    for (int m = 0; m < MR; m += 4) {
                        const float4 x4 = *reinterpret_cast<const float4 *>(xrow + m);
                        xv[m] = dup(x4.x * s); xv[m + 1] = dup(x4.y * s); xv[m + 2] = dup(x4.z * s); xv[m + 3] = dup(x4.w * s);
                    }
                } else {
                    #pragma unroll
                    for (int m = 0; m < MR; ++m) xv[m] = dup(xrow[m] * s);
                }
                xrow += kStep * XS;
                #pragma unroll
                for (int i = 0; i < kWords; ++i)
                    #pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        // {8 lane, byte q, 1, 0}: the entry's address
                        const uint32_t at = __byte_perm(codes[d][i], lane_word, 0x7604u | ((uint32_t)q << 4));
                        uint64_t w;
                        asm("ld.shared.b64 %0, [%1];" : "=l"(w) : "r"(at));
                        #pragma unroll
                        for (int m = 0; m < MR; ++m) fma2(acc[m][4 * i + q], w, xv[m]);
                    }
            };
            uint32_t i = 0;
            #pragma unroll 1
            for (; i + D <= steps; i += D) {
                #pragma unroll
                for (int d = 0; d < D; ++d) {
                    multiply(d);
                    fetch(d);
                }
            }
            #pragma unroll
            for (int d = 0; d < D; ++d)
                if (i + d < steps) multiply(d);  // (only in a segment's last piece: nothing left to ask for)
        }

        // ---- the segment's sums: lanes with the same columns, halving the columns a lane keeps ----
        float v[MR][8];
        #pragma unroll
        for (int m = 0; m < MR; ++m) {
            float a[CPL];
            #pragma unroll
            for (int i = 0; i < CPL / 2; ++i) unpack(acc[m][i], a[2 * i], a[2 * i + 1]);
            if constexpr (CPL == 32) {
                const bool up = lane & 16u;
                #pragma unroll
                for (int i = 0; i < 16; ++i)
                    a[i] = (up ? a[16 + i] : a[i]) + __shfl_xor_sync(0xffffffffu, up ? a[i] : a[16 + i], 16);
                const bool up8 = lane & 8u;
                #pragma unroll
                for (int i = 0; i < 8; ++i)
                    a[i] = (up8 ? a[8 + i] : a[i]) + __shfl_xor_sync(0xffffffffu, up8 ? a[i] : a[8 + i], 8);
            } else if constexpr (CPL == 16) {
                const bool up = lane & 16u;
                #pragma unroll
                for (int i = 0; i < 8; ++i)
                    a[i] = (up ? a[8 + i] : a[i]) + __shfl_xor_sync(0xffffffffu, up ? a[i] : a[8 + i], 16);
            }
            #pragma unroll
            for (int i = 0; i < 8; ++i) v[m][i] = a[i];
        }
        // group of eight columns this lane holds now, and the place of float4 q of a row in `red`
        const uint32_t group = CPL == 32 ? in_row * 4 + ((lane >> 4) & 1u) * 2 + ((lane >> 3) & 1u)
                               : CPL == 16 ? in_row * 2 + (lane >> 4) : lane;
        auto place = [](uint32_t q) { return q ^ ((q >> 3) & 7u); };
        const bool whole = !CLUSTER && b == 0 && e == p.units_per_strip;
        // (a CTA shares its first strip and its last one at most)
        float *slot = p.partial + (size_t)(2 * blockIdx.x + (u == u_begin ? 0 : 1)) * (MR * kStripCols);
        #pragma unroll
        for (int mg = 0; mg < MR; mg += MG) {
            __syncthreads();  // the sums of the rows before have been read
            #pragma unroll
            for (int m = 0; m < MG; ++m) {
                float4 *dst = reinterpret_cast<float4 *>(red + (warp * MG + m) * kStripCols);
                dst[place(2 * group)] = make_float4(v[mg + m][0], v[mg + m][1], v[mg + m][2], v[mg + m][3]);
                dst[place(2 * group + 1)] = make_float4(v[mg + m][4], v[mg + m][5], v[mg + m][6], v[mg + m][7]);
            }
            __syncthreads();
            for (uint32_t i = tid; i < MG * (kStripCols / 4); i += THREADS) {
                const uint32_t m = i / (kStripCols / 4), q = i % (kStripCols / 4);
                float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                #pragma unroll
                for (uint32_t w = 0; w < kWarps; ++w) {
                    const float4 o = reinterpret_cast<const float4 *>(red + (w * MG + m) * kStripCols)[place(q)];
                    s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
                }
                const uint32_t n = strip * kStripCols + 4 * q;
                if (CLUSTER) reinterpret_cast<float4 *>(xs + (mg + m) * kStripCols)[q] = s;  // (the activations have been used)
                else if (!whole) __stcg(reinterpret_cast<float4 *>(slot + (mg + m) * kStripCols) + q, s);
                else if (mg + m < p.rows && n < p.N) finish4(p, mg + m, n, s);
            }
        }
        if (CLUSTER) {
            // the cluster's sums, in the order of the parts; every CTA finishes a share of the outputs
            namespace cg = cooperative_groups;
            cg::cluster_group cluster = cg::this_cluster();
            const uint32_t part = cluster.block_rank();
            cluster.sync();
            for (uint32_t i = tid * p.parts + part; i < MR * (kStripCols / 4); i += THREADS * p.parts) {
                const uint32_t m = i / (kStripCols / 4), n = strip * kStripCols + 4 * (i % (kStripCols / 4));
                if (m >= p.rows || n >= p.N) continue;
                float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                #pragma unroll 4
                for (uint32_t c = 0; c < p.parts; ++c) {
                    const float4 o = reinterpret_cast<const float4 *>(cluster.map_shared_rank(xs, c))[i];
                    s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
                }
                finish4(p, m, n, s);
            }
            cluster.sync();  // nobody leaves while its sums are being read
            return;
        }
        if (!whole) {
            const uint32_t c0 = cta_of(strip * p.units_per_strip, p.total_units, ctas);
            const uint32_t c1 = cta_of((strip + 1) * p.units_per_strip - 1, p.total_units, ctas);
            __syncthreads();
            if (tid == 0) {
                __threadfence();
                const uint32_t sh = (strip & 3u) * 8u, parts = c1 - c0 + 1;
                uint32_t *counter = p.counters + (strip >> 2);
                const uint32_t old = (atomicAdd(counter, 1u << sh) >> sh) & 0xffu;
                if (old == parts - 1) atomicSub(counter, parts << sh);
                last_s = old == parts - 1 ? 1u : 0u;
            }
            __syncthreads();
            if (last_s) {
                __threadfence();
                // the parts of an output in order, split between threads where there are fewer outputs
                constexpr uint32_t kItems = MR * (kStripCols / 4), kGroups = kItems < THREADS ? THREADS / kItems : 1u;
                const uint32_t parts = c1 - c0 + 1, per = (parts + kGroups - 1) / kGroups;
                const uint32_t slot0 = 2 * c0 + (run_begin(p.total_units, c0, ctas) < strip * p.units_per_strip ? 1u : 0u);
                for (uint32_t i = tid; i < kItems * kGroups; i += THREADS) {
                    const uint32_t item = i % kItems, g = i / kItems;
                    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    #pragma unroll 8
                    for (uint32_t c = g * per; c < min(parts, (g + 1) * per); ++c) {
                        const size_t at = c == 0 ? slot0 : 2 * (size_t)(c0 + c);
                        const float4 o = __ldcg(reinterpret_cast<const float4 *>(p.partial + at * (MR * kStripCols)) + item);
                        s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
                    }
                    if (kGroups > 1) {
                        reinterpret_cast<float4 *>(red)[g * kItems + item] = s;
                    } else {
                        const uint32_t m = item / (kStripCols / 4), n = strip * kStripCols + 4 * (item % (kStripCols / 4));
                        if (m < p.rows && n < p.N) finish4(p, m, n, s);
                    }
                }
                if (kGroups > 1) {
                    __syncthreads();
                    if (tid < kItems) {
                        float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        #pragma unroll
                        for (uint32_t g = 0; g < kGroups; ++g) {
                            const float4 o = reinterpret_cast<const float4 *>(red)[g * kItems + tid];
                            s.x += o.x; s.y += o.y; s.z += o.z; s.w += o.w;
                        }
                        const uint32_t m = tid / (kStripCols / 4), n = strip * kStripCols + 4 * (tid % (kStripCols / 4));
                        if (m < p.rows && n < p.N) finish4(p, m, n, s);
                    }
                }
            }
        }
        u += e - b;
    }
    if (first) ptx::pdl_wait();  // (a CTA without work)
}

// T[m][j] = sum_k x[m][k] A(k, j), A [d_in][r] or [r][d_in]: a CTA per (m, j), eight warps share K, the
// warps' sums are added in warp order.
template <class T>
__global__ void __launch_bounds__(256)
strip_lora_t_kernel(const T *__restrict__ x, const T *__restrict__ a, float *__restrict__ t, uint32_t K, uint32_t rank, bool out_in) {
    __shared__ float part[8];
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t m = blockIdx.x / rank, j = blockIdx.x % rank;
    auto f = [](T v) { return (float)v; };
    float acc = 0.0f;
    #pragma unroll 8
    for (uint32_t k = threadIdx.x; k < K; k += 256)
        acc = fmaf(f(x[(size_t)m * K + k]), f(out_in ? a[(size_t)j * K + k] : a[(size_t)k * rank + j]), acc);
    #pragma unroll
    for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
    if (lane == 0) part[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        float v = 0.0f;
        #pragma unroll
        for (int w = 0; w < 8; ++w) v += part[w];
        t[(size_t)m * rank + j] = v;
    }
}

struct Runs {
    uint32_t ctas, units_per_strip, total;
    bool whole_strips;
};
// CTAs to a strip's cluster: 1 where runs over all strips are the better division.  A unit takes about 0.27 us at one row; a run's
// meeting through global memory costs six of them, the ends of the second segments where runs do not divide the strips evenly
// six more, a cluster's meeting four and half a unit for every CTA.  (More rows: longer units, and longer ends as well.)  1 x 4096 x 11008 15.7 -> 12.6 us in clusters of three, 1 x 512 x 11008 5.8 -> 5.0; in clusters of sixteen
// 1 x 4096 x 2048 went from 6.2 to 7.0.
uint32_t cluster_parts(const Runs &r, const ClusterRoom &room) {
    const uint32_t strips = r.total / r.units_per_strip;
    const uint32_t run = (r.total + r.ctas - 1) / r.ctas;
    const bool equal = r.total % r.ctas == 0, whole = equal && run % r.units_per_strip == 0, even = equal && r.units_per_strip % run == 0;
    uint32_t best = 1, least = run + (whole ? 0 : even ? 6 : 12);
    for (uint32_t c = 2; c <= 8 && c <= r.units_per_strip; ++c) {
        const uint32_t cost = (r.units_per_strip + c - 1) / c + 4 + c / 2;
        if (strips <= room.any[c] && strips * c <= persistent_ctas() && (cost < least || (cost == least && best > 1))) {
            least = cost;
            best = c;
        }
    }
    return best;
}
// A run keeps four units at least (256 rows of W: beyond that, what a strip's segments cost to meet
// outweighs the parallelism), and one CTA per SM at most.
bool deal_out(uint64_t K, uint64_t N, Runs &r) {
    if (N % kBlock != 0 || K == 0 || N == 0 || K >= (1ull << 30) || N >= (1ull << 30)) return false;
    const uint64_t strips = (N + kStripCols - 1) / kStripCols, ups = (K + kUnitRows - 1) / kUnitRows;
    if (strips * ups >= (1ull << 31)) return false;
    r.units_per_strip = (uint32_t)ups;
    r.total = (uint32_t)(strips * ups);
    r.whole_strips = strips > kCounterStrips;
    uint64_t ctas = r.total / 4;
    if (ctas > persistent_ctas()) ctas = persistent_ctas();
    if (ctas < 1) ctas = 1;
    r.ctas = (uint32_t)ctas;
    return true;
}

uint64_t up256(uint64_t v) { return (v + 255) / 256 * 256; }
uint32_t padded_rows(uint64_t rows) { return rows <= 1 ? 1 : rows <= 2 ? 2 : rows <= 4 ? 4 : rows <= 8 ? 8 : 16; }

template <int MR, int CPL, int THREADS, int D, bool DQ>
int32_t launch_as(StripParams &p, uint32_t ctas, cudaStream_t stream) {
    constexpr uint32_t kStep = THREADS / 32 * (32 / (kStripCols / CPL));
    p.x_rows = kXBytes / (4 * x_stride(MR)) / (D * kStep) * (D * kStep);
    const int smem = (int)(kTableAt + 0x10000 + kRedBytes - 1024);
    auto kernel = in_out_strip_kernel<MR, CPL, THREADS, D, DQ, true>;
    ClusterRoom room;
    NF4_TRY(cluster_room(reinterpret_cast<const void *>(kernel), THREADS, (uint32_t)smem, &room));
    Runs r;
    r.ctas = ctas;
    r.units_per_strip = p.units_per_strip;
    r.total = p.total_units;
    p.parts = cluster_parts(r, room);
    if (p.parts > 1) {
        ctas = p.total_units / p.units_per_strip * p.parts;
    } else {
        kernel = in_out_strip_kernel<MR, CPL, THREADS, D, DQ, false>;
        NF4_TRY(ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), smem));
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = p.parts;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = p.parts > 1 ? 2 : 1;
    count_launch();
    return check_cuda(cudaLaunchKernelEx(&cfg, kernel, p), "in_out_strip_kernel launch");
}

template <bool DQ>
int32_t launch(StripParams &p, uint32_t ctas, bool wide, cudaStream_t stream) {
    if (!wide) return p.rows <= 8 ? launch_as<8, 8, 512, 6, DQ>(p, ctas, stream) : launch_as<16, 8, 256, 6, DQ>(p, ctas, stream);
    switch (padded_rows(p.rows)) {
        case 1: return launch_as<1, 32, 512, 6, DQ>(p, ctas, stream);
        case 2: return launch_as<2, 16, 512, 8, DQ>(p, ctas, stream);
        case 4: return launch_as<4, 16, 512, 6, DQ>(p, ctas, stream);
        case 8: return launch_as<8, 8, 512, 6, DQ>(p, ctas, stream);
        default: return launch_as<16, 8, 256, 6, DQ>(p, ctas, stream);
    }
}

}  // namespace

int32_t small_lora_t(const void *x, const void *a, float *t, uint64_t rows, uint64_t K, uint32_t rank, bool f32, bool out_in, cudaStream_t stream) {
    const dim3 grid((unsigned)(rows * rank));
    count_launch();
    if (f32)
        return launch_maybe_overlapped(strip_lora_t_kernel<float>, grid, dim3(256), 0, stream, true, static_cast<const float *>(x),
                                       static_cast<const float *>(a), t, (uint32_t)K, rank, out_in);
    return launch_maybe_overlapped(strip_lora_t_kernel<__nv_bfloat16>, grid, dim3(256), 0, stream, true, static_cast<const __nv_bfloat16 *>(x),
                                   static_cast<const __nv_bfloat16 *>(a), t, (uint32_t)K, rank, out_in);
}

// flag words | T | two partial results per CTA (sized for sixteen rows where a call has more than one pass)
uint64_t strips_workspace_bytes(uint64_t rows, uint64_t d_in, uint64_t d_out, uint32_t lora_rank) {
    Runs r;
    if (rows == 0 || !deal_out(d_in, d_out, r)) return 0;
    const uint64_t mr = padded_rows(rows) < 8 ? 8 : padded_rows(rows);  // (codes at odd alignments run padded to eight rows)
    return 256 + up256(rows * lora_rank * 4) + (r.whole_strips ? 0 : 2ull * r.ctas * mr * kStripCols * 4);
}

bool strips_supported(const nf4_linear_args &a) {
    Runs r;
    return a.layout == NF4_LAYOUT_IN_OUT && deal_out(a.d_in, a.d_out, r) && (reinterpret_cast<uintptr_t>(a.packed) & 3u) == 0 &&
           a.workspace && a.workspace_bytes >= strips_workspace_bytes(a.rows, a.d_in, a.d_out, a.lora_a ? a.lora_rank : 0);
}

int32_t strips_forward(const nf4_linear_args &a, cudaStream_t stream) {
    Runs r;
    if (!strips_supported(a) || !deal_out(a.d_in, a.d_out, r)) return fail(NF4_ERR_UNSUPPORTED, "strips_forward: unsupported shape");
    const uint32_t rank = a.lora_a ? a.lora_rank : 0;
    uint8_t *ws = static_cast<uint8_t *>(a.workspace);
    float *t = reinterpret_cast<float *>(ws + 256);
    const bool f32 = a.io_dtype == NF4_DTYPE_F32;
    if (rank) NF4_TRY(small_lora_t(a.x, a.lora_a, t, a.rows, a.d_in, rank, f32, false, stream));
    const uint64_t ldy = a.ldy ? a.ldy : a.d_out;
    const size_t xb = f32 ? 4 : 2, yb = f32 || a.y_f32 ? 4 : 2;
    for (uint64_t m0 = 0; m0 < a.rows; m0 += 16) {  // sixteen activation rows per launch
        StripParams p{};
        p.x = static_cast<const uint8_t *>(a.x) + m0 * a.d_in * xb;
        p.y = static_cast<uint8_t *>(a.y) + m0 * ldy * yb;
        p.lora_b = a.lora_b;
        p.packed = a.packed;
        p.absmax = a.absmax;
        p.scale_codes = a.scale_codes;
        p.scale_of_scales = a.scale_of_scales;
        p.bias = a.bias;
        p.t = t + m0 * rank;
        p.counters = reinterpret_cast<uint32_t *>(ws);
        p.partial = reinterpret_cast<float *>(ws + 256 + up256(a.rows * rank * 4));
        p.rows = (uint32_t)(a.rows - m0 < 16 ? a.rows - m0 : 16);
        p.K = (uint32_t)a.d_in;
        p.N = (uint32_t)a.d_out;
        p.rank = rank;
        p.ldy = ldy;
        p.lora_scale = a.lora_scale;
        p.units_per_strip = r.units_per_strip;
        p.total_units = r.total;
        p.whole_strips = r.whole_strips;
        p.f32 = f32;
        p.y_f32 = (uint32_t)a.y_f32;
        p.y_vec = (reinterpret_cast<uintptr_t>(p.y) & (4 * yb - 1)) == 0 && ldy % 4 == 0;
        NF4_TRY(a.absmax ? launch<false>(p, r.ctas, aligned16(a.packed), stream) : launch<true>(p, r.ctas, aligned16(a.packed), stream));
    }
    return NF4_OK;
}

}  // namespace nf4
