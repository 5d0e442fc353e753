// What the tensor-core GEMM needs of the activations before it runs, and the adapter intermediate for
// the gradients: in one pass over x [M][K]
//   xh[m][k] = f16(x[m][k] / row_scale[m])  (row_scale: a power of two),
//   T = scale (x A^T) / row_scale as bf16 hi / lo halves (more k-steps of the GEMM),
//   R = x A^T likewise, unscaled (the operand of the gradient kernel).
//
// Split.  A cluster of CTAs takes 64 or 32 rows of x, each CTA a piece of K, which streams through shared
// memory in stages of 128 k (f32: 64) of x and of the adapter factor (16-byte asynchronous copies, two to five
// stages in flight): a stage is converted, written out and multiplied where it lies.  bf16 rows are nearly always
// converted as they are, so the copy does not wait for the row's maximum; a row that needs a power of
// two after all is written once more.  f32 rows need theirs first: x is read for the maxima, then (from L2) again.
// The CTAs' maxima and partial sums of T meet through distributed shared memory, in rank order
// (results do not depend on timing), after which each writes its share of the rows' T.  The factor
// [r][K] is the MMA's B operand as it lies, [K][r] goes through transposing matrix loads.
//
// Bound by the bytes of x in and xh out, and for few rows by the chain of a load, a stage and one exchange.  Pieces
// loaded whole, with an exchange of the maxima before anything was written and 32 rows to a factor tile, before:
// [2048, 4096] at rank 64 30 us, now 19; [2048, 14336] 93, now 52; product alone, [2048, 4096], 21, now 15.  f32 beside
// the repacking launch: the maxima are read while it runs, only the factor waits for it.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "kernels.cuh"
#include "ptx.cuh"

namespace nf4 {
namespace {

constexpr uint32_t kThreads = 256;
constexpr uint32_t kPartPitch = 68;  // floats
constexpr uint32_t kMaxCluster = 1u << (kClusterSizes - 1);
constexpr uint32_t kSmem = 108 * 1024;  // two CTAs on an SM
// A stage: 128 k of bf16, 64 of f32.  Pitches are 16 bytes off a multiple of 128 (conflict-free matrix loads), for
// the pairs of floats 32.
__host__ __device__ constexpr uint32_t stage_k(bool f32) { return f32 ? 64 : 128; }
__host__ __device__ constexpr uint32_t x_pitch(bool f32) { return f32 ? 288 : 272; }
__host__ __device__ constexpr uint32_t factor_pitch(bool f32, bool k_major) { return k_major || f32 ? 144 : 272; }
__host__ __device__ constexpr uint32_t factor_bytes(bool f32) { return (f32 ? 64 : 128) * 144; }  // the larger orientation
__host__ __device__ constexpr uint32_t stage_bytes(bool f32, uint32_t rows) { return rows * x_pitch(f32) + factor_bytes(f32); }
__host__ __device__ constexpr uint32_t stages_of(bool f32, uint32_t rows) { return kSmem / stage_bytes(f32, rows); }

struct Params {
    const void *x;
    const void *a;         // factor, bf16 (f16 for MODE 1)
    __half *xh;
    float *row_scale;
    __nv_bfloat16 *t_out, *r_out;  // [M][2 * 64 * chunks]: hi halves, then lo; or null
    const float *absmax;
    const uint8_t *scale_codes;
    const float *scale_of_scales;
    uint32_t *flags;
    uint32_t n_flags;
    uint32_t M, K, rank, chunks;
    uint32_t a_vec;        // the factor's rows are 16-byte aligned
    uint32_t piece;        // k per CTA, a multiple of 64
    float scale;
    uint32_t wait;         // for the kernel ahead: 0 first of all, 1 before the factor is read, 2 at the end
};

// Running maxima of |bf16|, a pair at a time (the sign bits mean nothing); a NaN leaves the maximum as
// it is (the operation returns the other operand).
__device__ __forceinline__ uint32_t bf16x2_absmax(uint32_t w, uint32_t mx) {
    uint32_t d;
    asm("max.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(w), "r"(mx));
    return d;
}
// The larger half of such a pair as an f32 pattern; 0 if only NaNs were seen.
__device__ __forceinline__ uint32_t bf16x2_larger_bits(uint32_t mx) {
    const uint32_t lo = (mx & 0x7fffu) << 16, hi = mx & 0x7fff0000u;
    const uint32_t a = lo <= 0x7f800000u ? lo : 0u, b = hi <= 0x7f800000u ? hi : 0u;
    return max(a, b);
}

__device__ __forceinline__ uint4 bf16x8_to_f16x8(const uint4 &v) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[4];
    #pragma unroll
    for (int q = 0; q < 4; ++q) {
        const __half2 h = __floats2half2_rn(__uint_as_float(w[q] << 16), __uint_as_float(w[q] & 0xffff0000u));
        o[q] = *reinterpret_cast<const uint32_t *>(&h);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}
__device__ __forceinline__ uint4 bf16x8_to_f16x8(const uint4 &v, float is) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t o[4];
    #pragma unroll
    for (int q = 0; q < 4; ++q) {
        const __half2 h = __floats2half2_rn(__uint_as_float(w[q] << 16) * is, __uint_as_float(w[q] & 0xffff0000u) * is);
        o[q] = *reinterpret_cast<const uint32_t *>(&h);
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

// The power of two a row is divided by.  bf16: only rows beyond f16's comfortable range (largest
// magnitude above 32768 or below 2^-8), brought to [16384, 32768); f32: every row.
template <bool F32>
__device__ __forceinline__ float row_factor(float mx) {
    const bool apply = F32 ? mx >= 1.1754944e-38f
                           : (mx > 32768.0f || (mx < 0.00390625f && mx >= 1.1754944e-38f)) && mx < __int_as_float(0x7f800000);
    if (!apply) return 1.0f;
    int e;
    frexpf(mx, &e);  // mx = f * 2^e with f in [0.5, 1)
    return ldexpf(1.0f, e - 15 < -100 ? -100 : e - 15);
}

// MODE 0: bf16 x (products with the bf16 factor are exact).  MODE 1: f32 x; the products use the scaled
// f16 copy and an f16 factor.  MODE 2: the product R alone, bf16.
template <int MODE, uint32_t kRows, bool k_major>
__global__ void __launch_bounds__(kThreads, 2)
prepass_kernel(const Params p) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    constexpr bool F32 = MODE == 1;
    constexpr uint32_t kStageK = stage_k(F32), kHalves = kStageK / 64;
    constexpr uint32_t kElem = F32 ? 4 : 2, kPitch = x_pitch(F32), kStage = stage_bytes(F32, kRows), kStages = stages_of(F32, kRows);
    constexpr uint32_t kRowTiles = kRows / 32;  // 16-row tiles of a warp
    static_assert(4 * kRows * kPartPitch * 4 <= kStages * kStage, "the sums reuse the stages");
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint32_t s_max[kMaxCluster][kRows];   // the CTAs' row maxima (f32 patterns)
    __shared__ float s_inv[kRows];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t cn = cluster.num_blocks(), rank_in = cluster.block_rank();
    const uint32_t m0 = (blockIdx.x / cn) * kRows, k0 = min(rank_in * p.piece, p.K), k1 = min(k0 + p.piece, p.K);
    const uint32_t base = ptx::smem_addr(smem);
    float *part = reinterpret_cast<float *>(smem);

    cluster.barrier_arrive();      // (waited for before the first access to another CTA's shared memory)
    // the GEMM may set itself up and start on the weights, which are in place once the kernels before this
    // one have completed (a repacked weight it waits for itself)
    if (p.wait == 0) ptx::pdl_wait();
    ptx::pdl_launch_dependents();
    // the GEMM's CTAs raise these once this kernel has completed (their readers and writers wait for that)
    if (blockIdx.x == 0)
        for (uint32_t i = tid; i < p.n_flags; i += kThreads) p.flags[i] = 0;

    const uint16_t *a = static_cast<const uint16_t *>(p.a);
    // A thread loads and converts k pieces of 8 (tid % 8 of every 64 k) of rows tid / 8, tid / 8 + 32 of a stage, and
    // loads the factor's likewise, 64 x 64 at a time.  Places and pointers are walked from stage to stage.
    const uint32_t tk = (tid & 7u) * 8, tr = tid >> 3;
    const uint8_t *xsrc[kRowTiles];
    const uint16_t *fsrc[2];
    uint32_t fsize[2], xsize[kRowTiles], next_k = 0, next_at = 0;
    auto start = [&](uint32_t chunk) {  // the loads from the first stage on, for the factor's 64 ranks `chunk`
        next_k = k0;
        next_at = base;
        #pragma unroll
        for (uint32_t q = 0; q < kRowTiles; ++q) {
            const bool real = m0 + tr + q * 32 < p.M;
            xsize[q] = real ? 16 : 0;
            xsrc[q] = static_cast<const uint8_t *>(p.x) + ((size_t)(real ? m0 + tr + q * 32 : 0) * p.K + k0 + tk) * kElem;
        }
        #pragma unroll
        for (uint32_t q = 0; q < 2; ++q) {
            const uint32_t r = tr + q * 32, j = chunk * 64 + (k_major ? tk : r);  // the rank; a row is a rank or a k
            fsize[q] = j < p.rank ? 16 : 0;
            fsrc[q] = k_major ? a + (size_t)(k0 + r) * p.rank + (fsize[q] ? j : 0) : a + (size_t)(fsize[q] ? j : 0) * p.K + k0 + tk;
        }
    };
    // The next stage; missing rows and ranks and the ragged end of K as zeros.
    auto load = [&](uint32_t chunk) {
        if (next_k < k1) {
            #pragma unroll
            for (uint32_t h = 0; h < kHalves; ++h) {
                const bool in = next_k + h * 64 + tk < k1;
                #pragma unroll
                for (uint32_t q = 0; q < kRowTiles; ++q) {
                    const uint32_t at = next_at + (tr + q * 32) * kPitch + (tk + h * 64) * kElem;
                    ptx::cp_async_16_or_zero(at, xsrc[q] + h * 64 * kElem, in ? xsize[q] : 0);
                    if (F32) ptx::cp_async_16_or_zero(at + 16, xsrc[q] + 16, in ? xsize[q] : 0);
                }
            }
            #pragma unroll
            for (uint32_t q = 0; q < kRowTiles; ++q) xsrc[q] += kStageK * kElem;
            const uint32_t fdst = next_at + kRows * kPitch;
            if (p.rank && p.a_vec) {
                #pragma unroll
                for (uint32_t h = 0; h < kHalves; ++h) {
                    #pragma unroll
                    for (uint32_t q = 0; q < 2; ++q) {
                        const uint32_t r = tr + q * 32;
                        const bool in = next_k + h * 64 + (k_major ? r : tk) < k1;
                        const uint32_t at = fdst + (k_major ? (r + h * 64) * 144 + tk * 2 : r * factor_pitch(F32, false) + (tk + h * 64) * 2);
                        ptx::cp_async_16_or_zero(at, fsrc[q] + h * (k_major ? 64 * p.rank : 64), in ? fsize[q] : 0);
                    }
                }
                #pragma unroll
                for (uint32_t q = 0; q < 2; ++q) fsrc[q] += k_major ? kStageK * p.rank : kStageK;
            } else if (p.rank) {  // rows at odd places: element by element
                for (uint32_t i = tid; i < 64 * kStageK; i += kThreads) {
                    const uint32_t c = k_major ? i & 63u : i % kStageK, r = k_major ? i >> 6 : i / kStageK;
                    const uint32_t k = next_k + (k_major ? r : c), j = chunk * 64 + (k_major ? c : r);
                    const uint16_t v = k < k1 && j < p.rank ? __ldg(a + (k_major ? (size_t)k * p.rank + j : (size_t)j * p.K + k)) : (uint16_t)0;
                    *reinterpret_cast<uint16_t *>(smem + (fdst - base) + r * factor_pitch(F32, k_major) + c * 2) = v;
                }
            }
            next_k += kStageK;
            next_at = next_at == base + (kStages - 1) * kStage ? base : next_at + kStage;
        }
        ptx::cp_async_commit();
    };
    auto begin = [&](uint32_t chunk) {
        start(chunk);
        for (uint32_t st = 0; st + 1 < kStages; ++st) load(chunk);
    };
    // The CTAs' maxima of a row -> its factor.  (Eight lanes hold a row's.)
    uint32_t mx[kRowTiles] = {};
    auto send_maxima = [&]() {
        #pragma unroll
        for (uint32_t q = 0; q < kRowTiles; ++q) {
            uint32_t m = F32 ? mx[q] : bf16x2_larger_bits(mx[q]);
            #pragma unroll
            for (int d = 1; d < 8; d *= 2) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
            for (uint32_t c = tid & 7u; c < cn; c += 8) cluster.map_shared_rank(&s_max[0][0], c)[rank_in * kRows + tr + q * 32] = m;
        }
    };
    auto factors = [&](int w_exp) {
        if (tid < kRows) {
            uint32_t m = 0;
            for (uint32_t c = 0; c < cn; ++c) m = max(m, s_max[c][tid]);
            const float sc = row_factor<F32>(__uint_as_float(m));
            s_inv[tid] = 1.0f / sc;  // exact: sc is a power of two
            if (rank_in == 0 && m0 + tid < p.M) p.row_scale[m0 + tid] = sc * ldexpf(1.0f, w_exp);  // both factors of the outputs
        }
        __syncthreads();
    };
    const int w_exp = MODE == 2 ? 0 : weight_exponent(p.absmax, p.scale_codes, p.scale_of_scales);

    if (F32) {
        #pragma unroll
        for (uint32_t q = 0; q < kRowTiles; ++q) {
            const uint32_t r = tr + q * 32;
            const float4 *row = reinterpret_cast<const float4 *>(static_cast<const float *>(p.x) + (size_t)(m0 + r) * p.K);
            if (m0 + r < p.M) {
                #pragma unroll 8
                for (uint32_t k = k0 / 4 + (tid & 7u); k < k1 / 4; k += 8) {
                    const float4 v = __ldg(row + k);
                    const uint32_t w[4] = {__float_as_uint(v.x), __float_as_uint(v.y), __float_as_uint(v.z), __float_as_uint(v.w)};
                    #pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if ((w[i] & 0x7fffffffu) < 0x7f800000u) mx[q] = max(mx[q], w[i] & 0x7fffffffu);
                }
            }
        }
        if (p.wait != 1) begin(0);
        cluster.barrier_wait();
        send_maxima();
        cluster.sync();
        factors(w_exp);
        if (p.wait == 1) {
            ptx::pdl_wait();
            begin(0);
        }
    } else {
        begin(0);
    }

    // ---- the stages: the f16 copy, and per stage a warp has half of the rows and 16 k, 64 ranks at a time ----
    const uint32_t rh = warp & 1u, kq = warp >> 1, g = lane >> 2, t = lane & 3u, li = lane >> 3, lr = lane & 7u;
    const float w_down = ldexpf(1.0f, -w_exp);
    const uint32_t per = kRows / cn, ld = 2 * 64 * p.chunks;
    constexpr uint32_t kSteps = kStageK / 64, kFactorPitch = factor_pitch(F32, k_major);  // 16 k each; of the factor's rows
    const uint32_t a_at = rh * kRowTiles * 16 * kPitch + ((li & 1u) * 8 + lr) * kPitch + (kq * kSteps * 16 + (li >> 1) * 8) * 2;
    const uint32_t b_at = kRows * kPitch + (k_major ? (kq * kSteps * 16 + (li & 1u) * 8 + lr) * kFactorPitch + (li >> 1) * 16
                                                    : ((li >> 1) * 8 + lr) * kFactorPitch + (kq * kSteps * 16 + (li & 1u) * 8) * 2);
    for (uint32_t chunk = 0; chunk < max(p.chunks, 1u); ++chunk) {
        float acc[kRowTiles][8][4] = {};
        const uint32_t tiles16 = p.rank ? (min(64u, p.rank - chunk * 64) + 15) / 16 : 0u;
        if (chunk) begin(chunk);
        uint32_t at = 0;  // the stage's place
        __half *out[kRowTiles];
        #pragma unroll
        for (uint32_t q = 0; q < kRowTiles; ++q) out[q] = p.xh + (size_t)(m0 + tr + q * 32) * p.K + k0 + tk;
        for (uint32_t ks = k0; ks < k1; ks += kStageK, at = at == (kStages - 1) * kStage ? 0 : at + kStage) {
            ptx::cp_async_wait<kStages - 2>();
            __syncthreads();
            load(chunk);
            if (MODE != 2 && chunk == 0) {
                #pragma unroll
                for (uint32_t q = 0; q < kRowTiles; ++q) {
                    const uint32_t r = tr + q * 32;
                    #pragma unroll
                    for (uint32_t h = 0; h < kHalves; ++h) {
                        const uint4 *in = reinterpret_cast<const uint4 *>(smem + at + r * kPitch + (tk + h * 64) * kElem);
                        uint4 o = in[0];
                        if (F32) {
                            const float is = s_inv[r];
                            const uint4 o2 = in[1];
                            const __half2 h0 = __floats2half2_rn(__uint_as_float(o.x) * is, __uint_as_float(o.y) * is);
                            const __half2 h1 = __floats2half2_rn(__uint_as_float(o.z) * is, __uint_as_float(o.w) * is);
                            const __half2 h2 = __floats2half2_rn(__uint_as_float(o2.x) * is, __uint_as_float(o2.y) * is);
                            const __half2 h3 = __floats2half2_rn(__uint_as_float(o2.z) * is, __uint_as_float(o2.w) * is);
                            o = make_uint4(*reinterpret_cast<const uint32_t *>(&h0), *reinterpret_cast<const uint32_t *>(&h1),
                                           *reinterpret_cast<const uint32_t *>(&h2), *reinterpret_cast<const uint32_t *>(&h3));
                        } else {
                            const uint32_t w[4] = {o.x, o.y, o.z, o.w};
                            #pragma unroll
                            for (int i = 0; i < 4; ++i) mx[q] = bf16x2_absmax(w[i], mx[q]);
                            o = bf16x8_to_f16x8(o);
                        }
                        if (m0 + r < p.M && ks + tk + h * 64 < k1) *reinterpret_cast<uint4 *>(out[q] + h * 64) = o;
                    }
                    out[q] += kStageK;
                }
            }
            if (!p.rank) continue;
            #pragma unroll
            for (uint32_t step = 0; step < kSteps; ++step) {
                uint32_t af[kRowTiles][4];
                #pragma unroll
                for (uint32_t q = 0; q < kRowTiles; ++q) {
                    if (F32) {
                        #pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint32_t r = (rh * kRowTiles + q) * 16 + g + (i & 1) * 8;
                            const float2 f = *reinterpret_cast<const float2 *>(smem + at + r * kPitch + (kq * 16 + 2 * t + (i >> 1) * 8) * 4);
                            const float is = s_inv[r];
                            const __half2 h = __floats2half2_rn(f.x * is, f.y * is);
                            af[q][i] = *reinterpret_cast<const uint32_t *>(&h);
                        }
                    } else {
                        ptx::ldmatrix_x4(af[q], base + at + a_at + q * 16 * kPitch + step * 32);
                    }
                }
                #pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    if (u >= tiles16) break;
                    uint32_t bf[4];
                    if (k_major) ptx::ldmatrix_x4_trans(bf, base + at + b_at + u * 32 + step * 16 * kFactorPitch);
                    else ptx::ldmatrix_x4(bf, base + at + b_at + u * 16 * kFactorPitch + step * 32);
                    #pragma unroll
                    for (uint32_t q = 0; q < kRowTiles; ++q) {
                        if (F32) {
                            ptx::mma_16816_f16(acc[q][2 * u], af[q][0], af[q][1], af[q][2], af[q][3], bf[0], bf[1]);
                            ptx::mma_16816_f16(acc[q][2 * u + 1], af[q][0], af[q][1], af[q][2], af[q][3], bf[2], bf[3]);
                        } else {
                            ptx::mma_16816_bf16(acc[q][2 * u], af[q][0], af[q][1], af[q][2], af[q][3], bf[0], bf[1]);
                            ptx::mma_16816_bf16(acc[q][2 * u + 1], af[q][0], af[q][1], af[q][2], af[q][3], bf[2], bf[3]);
                        }
                    }
                }
            }
        }
        ptx::cp_async_wait<0>();
        if (p.rank) {
            // the four k-quarters of the CTA add up in order, in the first one's place
            __syncthreads();
            #pragma unroll
            for (uint32_t q = 0; q < kRowTiles; ++q) {
                float *lo = part + ((kq * kRows) + (rh * kRowTiles + q) * 16 + g) * kPartPitch + 2 * t;
                #pragma unroll
                for (int u = 0; u < 8; ++u) {
                    *reinterpret_cast<float2 *>(lo + 8 * u) = make_float2(acc[q][u][0], acc[q][u][1]);
                    *reinterpret_cast<float2 *>(lo + 8 * kPartPitch + 8 * u) = make_float2(acc[q][u][2], acc[q][u][3]);
                }
            }
            __syncthreads();
            for (uint32_t i = tid; i < kRows * 16; i += kThreads) {
                float4 *at = reinterpret_cast<float4 *>(part + (i >> 4) * kPartPitch + (i & 15u) * 4);
                float4 v = *at;
                #pragma unroll
                for (uint32_t q = 1; q < 4; ++q) {
                    const float4 w = at[q * kRows * (kPartPitch / 4)];
                    v = make_float4(v.x + w.x, v.y + w.y, v.z + w.z, v.w + w.w);
                }
                *at = v;
            }
        }
        if (chunk == 0 && !F32) {
            cluster.barrier_wait();
            if (MODE == 0) send_maxima();
        }
        cluster.sync();
        if (chunk == 0 && MODE == 0) {
            factors(w_exp);
            for (uint32_t r = warp; r < kRows; r += kThreads / 32) {  // the rare rows with a factor, again
                const float is = s_inv[r];
                if (is == 1.0f || m0 + r >= p.M) continue;
                for (uint32_t k = k0 + lane * 8; k < k1; k += 256) {
                    const size_t at = (size_t)(m0 + r) * p.K + k;
                    *reinterpret_cast<uint4 *>(p.xh + at) = bf16x8_to_f16x8(__ldg(reinterpret_cast<const uint4 *>(static_cast<const uint16_t *>(p.x) + at)), is);
                }
            }
        }
        if (!p.rank) break;
        for (uint32_t i = tid; i < per * 16; i += kThreads) {
            const uint32_t r = rank_in * per + (i >> 4), c = (i & 15u) * 4, m = m0 + r;
            float sum[4] = {};
            #pragma unroll 4
            for (uint32_t q = 0; q < cn; ++q) {
                const float4 w = *reinterpret_cast<const float4 *>(cluster.map_shared_rank(part, q) + r * kPartPitch + c);
                sum[0] += w.x;
                sum[1] += w.y;
                sum[2] += w.z;
                sum[3] += w.w;
            }
            if (m >= p.M) continue;
            const size_t at = (size_t)m * ld + chunk * 64 + c;
            auto put = [&](__nv_bfloat16 *out, float f) {
                uint32_t hi[2], lo[2];
                #pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float v0 = sum[2 * h] * f, v1 = sum[2 * h + 1] * f;
                    const __nv_bfloat162 b = __floats2bfloat162_rn(v0, v1);
                    const __nv_bfloat162 l = __floats2bfloat162_rn(v0 - __low2float(b), v1 - __high2float(b));
                    hi[h] = *reinterpret_cast<const uint32_t *>(&b);
                    lo[h] = *reinterpret_cast<const uint32_t *>(&l);
                }
                *reinterpret_cast<uint2 *>(out + at) = make_uint2(hi[0], hi[1]);
                *reinterpret_cast<uint2 *>(out + at + 64 * p.chunks) = make_uint2(lo[0], lo[1]);
            };
            // (MODE 1: the products were taken with the scaled rows)
            if (MODE != 2) put(p.t_out, F32 ? p.scale * w_down : p.scale * s_inv[r] * w_down);
            if (MODE == 2 || p.r_out) put(p.r_out, 1.0f);
        }
        cluster.sync();  // the sums have been read (before the next chunk's stages, and before a CTA leaves)
    }
    if (p.wait == 2) ptx::pdl_wait();
}

}  // namespace

int32_t activations_prepass(const PrepassArgs &q, cudaStream_t stream) {
    Params p{};
    p.x = q.x;
    p.a = q.a;
    p.xh = static_cast<__half *>(q.xh);
    p.row_scale = q.row_scale;
    p.t_out = static_cast<__nv_bfloat16 *>(q.t_out);
    p.r_out = static_cast<__nv_bfloat16 *>(q.r_out);
    p.absmax = q.absmax;
    p.scale_codes = q.scale_codes;
    p.scale_of_scales = q.scale_of_scales;
    p.flags = q.flags;
    p.n_flags = q.n_flags;
    p.M = q.M;
    p.K = q.K;
    p.rank = q.rank;
    p.chunks = (q.rank + 63) / 64;
    p.a_vec = aligned16(q.a) && (q.k_major ? q.rank : q.K) % 8 == 0;
    p.scale = q.scale;
    p.wait = !q.beside_predecessor ? 0 : q.factor_of_predecessor ? 1 : 2;
    // 64 rows to a cluster beyond 512 rows, where the clusters of 32 no longer fit the chip at once, else 32 (half of the
    // factor's traffic against more CTAs)
    const uint32_t rows = q.M > 512 ? 64 : 32;
    const uint64_t tiles = (q.M + rows - 1) / rows;
    auto pick = [&](auto km) {
        constexpr bool k_major = decltype(km)::value;
        return rows == 64 ? (q.xh ? prepass_kernel<0, 64, k_major> : prepass_kernel<2, 64, k_major>)
                          : (q.xh ? prepass_kernel<0, 32, k_major> : prepass_kernel<2, 32, k_major>);
    };
    if (q.x_f32 && q.k_major) return fail(NF4_ERR_UNSUPPORTED, "activations_prepass: f32 factors come as [r][K]");
    auto kernel = q.x_f32 ? (rows == 64 ? prepass_kernel<1, 64, false> : prepass_kernel<1, 32, false>)
                          : q.k_major ? pick(std::true_type{}) : pick(std::false_type{});
    const int smem = (int)(stages_of(q.x_f32, rows) * stage_bytes(q.x_f32, rows));
    // as many CTAs of K as the chip holds at once, two on an SM (a second wave took 21 us where one takes 11)
    ClusterRoom room;
    NF4_TRY(cluster_room(reinterpret_cast<const void *>(kernel), kThreads, (uint32_t)smem, &room));
    const uint32_t cn = cluster_ctas(tiles, q.K, 64, room);
    p.piece = ((q.K + cn - 1) / cn + 63) / 64 * 64;
    if (tiles * cn >= (1ull << 31)) return fail(NF4_ERR_UNSUPPORTED, "activations_prepass: too many rows");
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(tiles * cn));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cn;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    count_launch();
    return check_cuda(cudaLaunchKernelEx(&cfg, kernel, p), "prepass_kernel launch");
}

}  // namespace nf4
