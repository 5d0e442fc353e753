// Shared device/host helpers of the NF4 B200 library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/nf4_b200.h"
#include "nf4_tables.inc"

namespace nf4 {

constexpr int kBlock = NF4_BLOCK_SIZE;  // values per quantization block
constexpr int kNumSMs = 148;            // B200

// ---- error plumbing (defined in api.cu) ------------------------------------
int32_t fail(int32_t code, const char *fmt, ...);
int32_t check_cuda(cudaError_t e, const char *what);
void count_launch(uint64_t n = 1);

#define NF4_CUDA_TRY(expr)                                         \
    do {                                                           \
        int32_t _st = ::nf4::check_cuda((expr), #expr);            \
        if (_st != NF4_OK) return _st;                             \
    } while (0)

#define NF4_TRY(expr)                  \
    do {                               \
        int32_t _st = (expr);          \
        if (_st != NF4_OK) return _st; \
    } while (0)

// ---- tables -----------------------------------------------------------------
static __device__ __constant__ const uint32_t c_level_bits[16] = {NF4_LEVEL_BITS_LIST};
// the same levels rounded to f16 (bit patterns)
static __device__ __constant__ const uint32_t c_level_f16_bits[16] = {NF4_LEVEL_F16_BITS_LIST};
static const uint32_t h_level_bits[16] = {NF4_LEVEL_BITS_LIST};
static const uint32_t h_threshold_bits[15] = {NF4_THRESHOLD_BITS_LIST};

// Decision thresholds as compile-time immediates (bit patterns from nf4_tables.inc).
struct ThresholdBits {
    uint32_t t[15];
};
__host__ __device__ constexpr ThresholdBits threshold_bits() { return {{NF4_THRESHOLD_BITS_LIST}}; }

template <int I>
__device__ __forceinline__ float T() {
    constexpr ThresholdBits tb = threshold_bits();
    return __uint_as_float(tb.t[I]);
}

// Code of an already-normalised value.  Equals the reference's sixteen-way scan
// (strict '<', lower index on ties) for NaN (code 0) and for every v with
// |v| <= 65536: there the scan's answer is the number of thresholds T_i with
// v >= T_i, found here by a four-step bisection on immediates.  (For much larger |v|
// the f32 differences v - L_i collapse onto each other and the scan drifts back to
// code 0; the quantizer never gets there, because |x| <= absmax makes
// |x / absmax| <= 1 and inf / inf is NaN.)
__device__ __forceinline__ uint32_t code_of_normalized(float v) {
    const bool b3 = v >= T<7>();
    const float t2 = b3 ? T<11>() : T<3>();
    const bool b2 = v >= t2;
    const float t1 = b3 ? (b2 ? T<13>() : T<9>()) : (b2 ? T<5>() : T<1>());
    const bool b1 = v >= t1;
    const float t0hi = b2 ? (b1 ? T<14>() : T<12>()) : (b1 ? T<10>() : T<8>());
    const float t0lo = b2 ? (b1 ? T<6>() : T<4>()) : (b1 ? T<2>() : T<0>());
    const float t0 = b3 ? t0hi : t0lo;
    const bool b0 = v >= t0;
    return (b3 ? 8u : 0u) | (b2 ? 4u : 0u) | (b1 ? 2u : 0u) | (b0 ? 1u : 0u);
}

// The reference's literal scan; used by the self-check kernel only.
__device__ __forceinline__ uint32_t code_by_scan(float v) {
    uint32_t best = 0;
    float best_dist = __int_as_float(0x7f800000);
    #pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float d = fabsf(__fsub_rn(v, __uint_as_float(c_level_bits[i])));
        if (d < best_dist) {
            best_dist = d;
            best = i;
        }
    }
    return best;
}

// Code of one raw value given its block's absmax (src/quantize.rs:109-112).
__device__ __forceinline__ uint32_t code_of(float x, float absmax) {
    if (absmax == 0.0f) return 7u;  // nearest level to 0.0
    return code_of_normalized(__fdiv_rn(x, absmax));
}

// ---- fast code selection ------------------------------------------------------------------
// One word per cell of width 1/16 over [-1, 1] (gen_nf4_tables.py): the only decision threshold that
// can lie in the cell and the number of thresholds below it, in the form FastCodes subtracts.
constexpr int kCellWords = 64;  // padded: any masked index is inside
static __device__ __constant__ const uint32_t c_cell_table[kCellWords] = {NF4_CELL_TABLE_LIST};

// Out of line on purpose: taken for a few values in a million, and inlining sixteen copies of
// the division and the bisection doubles the quantize kernel's register count.
static __device__ __noinline__ uint32_t code_of_exact(float x, float absmax) { return code_of(x, absmax); }

// Codes of up to eight values x / absmax without the division, where that is provably safe.
//   u = bits of fma(x, 2^21 rcp, 1.5 * 2^23) = 0x4b400000 + the quotient in units of 2^-21, with rcp the
//   hardware's reciprocal (within one ulp): within 0.88 units of the correctly rounded quotient (half
//   for the rounding to units, a quarter for rcp, an eighth for the quotient; |x| <= absmax).  A second multiply-add leaves 4 * cell of the quotient in the low bits of its
//   result; the cell's word W holds the only threshold that can matter and the count of those below,
//   so that u - W has the code in its top four bits.  Unless the low 28 bits say that the quotient is
//   within NF4_CELL_MARGIN (2) units of that threshold (rounded to units), the exact quotient is on the
//   same side of it.
//   Otherwise -- or for a NaN, or a scale outside [1e-30, 1e30] where rcp is not trustworthy -- the
//   caller decides every value of the group with code_of_exact.  No threshold is within 1e-4 of a
//   cell's edge, so it does not matter which of two neighbouring cells a value at an edge is given to.
// What it costs.  Instruction issue bounds a quantizer that is not bound by memory, and the integer
// pipe has half the rate of the FMA pipe: per value two multiply-adds, a mask, the table load, a
// subtraction, a funnel shift that collects the code, and a mask and minimum for the nearest threshold;
// 22 instructions per value with a conversion, a clamp and selects, 18 with a compare per threshold in f32.
// `cells` is the table in shared memory (a bank per cell: no conflicts).
struct FastCodes {
    uint32_t codes = 0, nearest = 0xffffffffu;

    // values are taken from the last (highest nibble) to the first; rcp = approx_rcp(absmax)
    __device__ __forceinline__ void take(float x, float rcp_units, float rcp_cells, const uint32_t *cells) {
        const uint32_t u = __float_as_uint(fmaf(x, rcp_units, 12582912.0f));
        const uint32_t at = __float_as_uint(fmaf(x, rcp_cells, 12582912.0f + 64.0f)) & 0xfcu;
        const uint32_t d = u - *reinterpret_cast<const uint32_t *>(reinterpret_cast<const char *>(cells) + at);
        codes = __funnelshift_l(d, codes, 4);
        nearest = min(nearest, d & 0x0fffffffu);
    }
    __device__ __forceinline__ bool sure() const { return nearest >= 2u * NF4_CELL_MARGIN; }
};

__device__ __forceinline__ float approx_rcp(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// The eight codes of a group as nibbles, the first value in the lowest.
__device__ __forceinline__ uint32_t codes_of_group(const float (&x)[8], float absmax, const uint32_t *cells) {
    const float rcp = approx_rcp(absmax);
    FastCodes f;
    #pragma unroll
    for (int i = 7; i >= 0; --i) f.take(x[i], rcp * 2097152.0f, rcp * 64.0f, cells);
    uint32_t w = f.codes;
    if (!f.sure() || !(absmax >= 1e-30f && absmax <= 1e30f)) {
        w = 0;
        #pragma unroll
        for (int i = 0; i < 8; ++i) w |= code_of_exact(x[i], absmax) << (4 * i);
    }
    return w;
}

// The same for eight bf16 values of a block whose scale is in [1e-30, 1e30], none of them a NaN: the quotients of two bf16
// numbers leave gaps around the thresholds that are wider than the approximation's error, the cuts of `cells`
// (c_cell_bf16_table) lie in their middle, and nothing is left to decide otherwise.
static __device__ __constant__ const uint32_t c_cell_bf16_table[kCellWords] = {NF4_CELL_BF16_TABLE_LIST};
__device__ __forceinline__ uint32_t codes_of_bf16(const float (&x)[8], float rcp_units, float rcp_cells, const uint32_t *cells) {
    uint32_t codes = 0;
    #pragma unroll
    for (int i = 7; i >= 0; --i) {
        const uint32_t u = __float_as_uint(fmaf(x[i], rcp_units, 12582912.0f));
        const uint32_t at = __float_as_uint(fmaf(x[i], rcp_cells, 12582912.0f + 64.0f)) & 0xfcu;
        codes = __funnelshift_l(u - *reinterpret_cast<const uint32_t *>(reinterpret_cast<const char *>(cells) + at), codes, 4);
    }
    return codes;
}

// Scale of a double-quantized block: divide first, then multiply (src/quantize.rs:348).
__device__ __forceinline__ float dq_scale(uint32_t code, float scale_of_scales) {
    return __fmul_rn(__fdiv_rn((float)code, 255.0f), scale_of_scales);
}

// The tensor-core GEMM scales the expanded levels in f16, so block scales must sit inside f16's
// normal range (6.1e-5 .. 65504).  It and its pre-pass therefore work with scales divided by 2^e, e the
// exponent of the weight's first block scale (the scales of one weight lie within a few powers of
// two of each other), and the outputs are multiplied back by 2^e: the pre-pass folds 2^e into the
// rows' factors and 2^-e into the adapter intermediate.  Powers of two: every step is exact.
__device__ __forceinline__ int weight_exponent(const float *absmax, const uint8_t *scale_codes,
                                               const float *scale_of_scales) {
    const float s0 = absmax ? __ldg(absmax) : dq_scale(__ldg(scale_codes), __ldg(scale_of_scales));
    if (!(s0 > 0.0f) || s0 >= __int_as_float(0x7f800000)) return 0;
    int e;
    frexpf(s0, &e);  // s0 = f * 2^e, f in [0.5, 1)
    return min(max(e, -100), 100);
}

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace nf4
