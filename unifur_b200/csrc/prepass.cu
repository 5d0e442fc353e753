// What the tensor-core GEMM needs of the activations before it runs, and the adapter intermediate for
// the gradients: in one pass over x [M][K]
//   xh[m][k] = f16(x[m][k] / row_scale[m])  (row_scale: a power of two),
//   T = scale (x A^T) / row_scale as bf16 hi / lo halves (more k-steps of the GEMM),
//   R = x A^T likewise, unscaled (the operand of the gradient kernel).
//
// Split.  A cluster of CTAs takes 64 or 32 rows of x, each CTA a piece of K, which streams through shared
// memory in stages of 128 k of x and of the adapter factor (16-byte asynchronous copies, two or three
// stages in flight): a stage is converted, written out and multiplied where it lies.  bf16 rows are nearly always
// converted as they are, so the copy does not wait for the row's maximum; a row that needs a power of
// two after all is written once more.  (f32 rows need theirs first: a kernel of their own below.)
// The CTAs' maxima and partial sums of T meet through distributed shared memory, in rank order
// (results do not depend on timing), after which each writes its share of the rows' T.  The factor
// [r][K] is the MMA's B operand as it lies, [K][r] goes through transposing matrix loads.
//
// Bound by the bytes of x in and xh out, and for few rows by the chain of a load, a stage and one exchange.  Pieces
// loaded whole, with an exchange of the maxima before anything was written and 32 rows to a factor tile, before:
// [2048, 4096] at rank 64 30 us, now 19; [2048, 14336] 93, now 52; product alone, [2048, 4096], 21, now 15.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <type_traits>

#include "kernels.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace nf4 {
namespace {

constexpr uint32_t kThreads = 256;
constexpr uint32_t kPartPitch = 68;  // floats
constexpr uint32_t kMaxCluster = 1u << (kClusterSizes - 1);
constexpr uint32_t kSmem = 108 * 1024;  // two CTAs on an SM
// A stage: 128 k.  Pitches are 16 bytes off a multiple of 128 (conflict-free matrix loads).
constexpr uint32_t kStageK = 128, kPitch = 272;
__host__ __device__ constexpr uint32_t factor_pitch(bool k_major) { return k_major ? 144 : 272; }
constexpr uint32_t kFactorBytes = 128 * 144;  // the larger orientation
__host__ __device__ constexpr uint32_t stage_bytes(uint32_t rows) { return rows * kPitch + kFactorBytes; }
__host__ __device__ constexpr uint32_t stages_of(uint32_t rows) { return kSmem / stage_bytes(rows); }

struct Params {
    const void *x;
    const void *a;         // factor, of x's type
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

// Running minima of the nonzero |bf16|, a pair at a time, as patterns one or two below them: taking one off turns a zero into
// a NaN, which the minimum leaves out.  (A zero's borrow reaches the upper half, where it may make a NaN of the smallest
// subnormal; no power of two used here brings that one into f16's range.)
__device__ __forceinline__ uint32_t bf16x2_absmin(uint32_t w, uint32_t mn) {
    uint32_t d;
    asm("min.xorsign.abs.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(w - 0x00010001u), "r"(mn));
    return d;
}
// What was seen of a row as one word: its largest value above the negative of its least nonzero one (infinity: it has none),
// both as bf16, so that words join by one maximum of pairs.
__device__ __forceinline__ uint32_t row_seen(uint32_t mx, uint32_t mn) {
    return bf16x2_larger_bits(mx) | 0x8000u | min(min(mn & 0x7fffu, (mn >> 16) & 0x7fffu), 0x7f80u);
}
__device__ __forceinline__ uint32_t join_seen(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
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

// Four sums times f as bf16 high halves at out[at], low halves `lo` elements on; out may be null.
__device__ __forceinline__ void put_halves(__nv_bfloat16 *out, const float (&sum)[4], float f, size_t at, uint32_t lo) {
    if (!out) return;
    uint32_t hi[2], low[2];
    #pragma unroll
    for (int h = 0; h < 2; ++h) {
        const float v0 = sum[2 * h] * f, v1 = sum[2 * h + 1] * f;
        const __nv_bfloat162 b = __floats2bfloat162_rn(v0, v1);
        const __nv_bfloat162 l = __floats2bfloat162_rn(v0 - __low2float(b), v1 - __high2float(b));
        hi[h] = *reinterpret_cast<const uint32_t *>(&b);
        low[h] = *reinterpret_cast<const uint32_t *>(&l);
    }
    *reinterpret_cast<uint2 *>(out + at) = make_uint2(hi[0], hi[1]);
    *reinterpret_cast<uint2 *>(out + at + lo) = make_uint2(low[0], low[1]);
}

// bf16 x (products with the bf16 factor are exact).  MODE 0: the copy, and T (or R).  MODE 2: the product R alone.
template <int MODE, uint32_t kRows, bool k_major>
__global__ void __launch_bounds__(kThreads, 2)
prepass_kernel(const Params p) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    constexpr uint32_t kHalves = kStageK / 64, kElem = 2, kStage = stage_bytes(kRows), kStages = stages_of(kRows);
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
    ptx::pdl_wait();
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
                        const uint32_t at = fdst + (k_major ? (r + h * 64) * 144 + tk * 2 : r * factor_pitch(false) + (tk + h * 64) * 2);
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
                    *reinterpret_cast<uint16_t *>(smem + (fdst - base) + r * factor_pitch(k_major) + c * 2) = v;
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
            uint32_t m = bf16x2_larger_bits(mx[q]);
            #pragma unroll
            for (int d = 1; d < 8; d *= 2) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
            for (uint32_t c = tid & 7u; c < cn; c += 8) cluster.map_shared_rank(&s_max[0][0], c)[rank_in * kRows + tr + q * 32] = m;
        }
    };
    auto factors = [&](int w_exp) {
        if (tid < kRows) {
            uint32_t m = 0;
            for (uint32_t c = 0; c < cn; ++c) m = max(m, s_max[c][tid]);
            const float sc = row_factor<false>(__uint_as_float(m));
            s_inv[tid] = 1.0f / sc;  // exact: sc is a power of two
            if (rank_in == 0 && m0 + tid < p.M) p.row_scale[m0 + tid] = sc * ldexpf(1.0f, w_exp);  // both factors of the outputs
        }
        __syncthreads();
    };
    const int w_exp = MODE == 2 ? 0 : weight_exponent(p.absmax, p.scale_codes, p.scale_of_scales);

    begin(0);

    // ---- the stages: the f16 copy, and per stage a warp has half of the rows and 16 k, 64 ranks at a time ----
    const uint32_t rh = warp & 1u, kq = warp >> 1, g = lane >> 2, t = lane & 3u, li = lane >> 3, lr = lane & 7u;
    const float w_down = ldexpf(1.0f, -w_exp);
    const uint32_t per = kRows / cn, ld = 2 * 64 * p.chunks;
    constexpr uint32_t kSteps = kStageK / 64, kFactorPitch = factor_pitch(k_major);  // 16 k each; of the factor's rows
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
                        const uint32_t w[4] = {o.x, o.y, o.z, o.w};
                        #pragma unroll
                        for (int i = 0; i < 4; ++i) mx[q] = bf16x2_absmax(w[i], mx[q]);
                        o = bf16x8_to_f16x8(o);
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
                    ptx::ldmatrix_x4(af[q], base + at + a_at + q * 16 * kPitch + step * 32);
                }
                #pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    if (u >= tiles16) break;
                    uint32_t bf[4];
                    if (k_major) ptx::ldmatrix_x4_trans(bf, base + at + b_at + u * 32 + step * 16 * kFactorPitch);
                    else ptx::ldmatrix_x4(bf, base + at + b_at + u * 16 * kFactorPitch + step * 32);
                    #pragma unroll
                    for (uint32_t q = 0; q < kRowTiles; ++q) {
                        ptx::mma_16816_bf16(acc[q][2 * u], af[q][0], af[q][1], af[q][2], af[q][3], bf[0], bf[1]);
                        ptx::mma_16816_bf16(acc[q][2 * u + 1], af[q][0], af[q][1], af[q][2], af[q][3], bf[2], bf[3]);
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
        if (chunk == 0) {
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
            if (MODE != 2) put_halves(p.t_out, sum, p.scale * s_inv[r] * w_down, at, 64 * p.chunks);
            put_halves(p.r_out, sum, 1.0f, at, 64 * p.chunks);
        }
        cluster.sync();  // the sums have been read (before the next chunk's stages, and before a CTA leaves)
    }
}

// ---- f32 x ------------------------------------------------------------------------------------------------------------
// T's products use the scaled f16 copy and the factor rounded to f16.  A cluster takes 32 rows, a CTA a piece of K: 32 k
// at a time a warp, whose lanes hold eight k of four rows each, as the MMA's A operand wants them (in an order of k
// that the factor's lanes share).  Up to 512 k, the usual case, the values stay in registers while the rows' maxima meet, so that x
// is read once, all of it in flight together, and the factor's values are on their way beside it; of longer pieces all but the last 512 k are read again.
// The factor comes as it is stored, f32 in either orientation.  T appears twice, in columns j and rank + j: the GEMM
// multiplies it with the bf16 high and low halves of the other factor.
// Bound by the chain of the loads, the maxima's exchange, the copy and the sums' exchange.  Before, with x read twice (the
// second time behind the exchange, through shared memory) and a launch ahead that converted both factors, the two took 14 us of
// the 42.2 of 512 x 4096 x 4096 at rank 16; now 9 of 33.1.  [2048, 4096] at rank 64 43 us and 6 for the factors, now 31;
// [4096, 14336] at rank 8 133 and 6, now 124.  (The copy with a factor from the row's first values, without the maxima's
// exchange, and T in tf32 from registers, both factors converted where they are used: 512 x 4096 x 4096 36.9
// where the present way took 32.6.)
constexpr uint32_t kUnits = 2, kPieceF32 = 8 * kUnits * 32, kGroupRanks = 16, kMostRanks = 128, kPartRow = 20, kSumRow = kMostRanks + 4;

template <bool k_major>
__global__ void __launch_bounds__(kThreads, 2)
prepass_f32_kernel(const Params p) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    constexpr uint32_t kRows = 32;
    __shared__ uint32_t s_warp[8][kRows], s_max[kMaxCluster][kRows];  // row maxima: of the warps, of the CTAs (f32 patterns)
    __shared__ float s_inv[kRows];
    __shared__ __align__(16) float s_part[8][kRows][kPartRow];  // the warps' sums of sixteen ranks
    __shared__ __align__(16) float s_sum[kRows][kSumRow];       // this CTA's of all
    extern __shared__ __align__(16) float s_all[];              // the CTAs', of this one's share of the rows [cn][32 / cn][kSumRow]
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, g = lane >> 2, t = lane & 3u;
    const uint32_t cn = cluster.num_blocks(), rank_in = cluster.block_rank();
    const uint32_t m0 = (blockIdx.x / cn) * kRows, k0 = min(rank_in * p.piece, p.K), k1 = min(k0 + p.piece, p.K);

    ptx::pdl_wait();
    ptx::pdl_launch_dependents();  // (what for: see the kernel above)
    cluster.barrier_arrive();  // (waited for before the first access to another CTA's shared memory)
    if (blockIdx.x == 0)
        for (uint32_t i = tid; i < p.n_flags; i += kThreads) p.flags[i] = 0;

    // A lane's values of a unit of 32 k: rows q * 8 + g, k 16 s + 4 t and the three after it (K and the pieces are
    // multiples of 64: a unit is whole or empty).
    float4 v[kUnits][4][2];
    auto load = [&](uint32_t kp) {
        #pragma unroll
        for (uint32_t u = 0; u < kUnits; ++u) {
            const uint32_t k = kp + (u * 8 + warp) * 32 + 4 * t;
            #pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                const uint32_t m = m0 + q * 8 + g;
                const float4 *src = reinterpret_cast<const float4 *>(static_cast<const float *>(p.x) + (size_t)m * p.K + k);
                const bool in = m < p.M && k < k1;
                #pragma unroll
                for (uint32_t s = 0; s < 2; ++s) v[u][q][s] = in ? __ldg(src + 4 * s) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            }
        }
    };
    // The factor's values of the same k, ranks group * 16 + 8 n + g, as the MMA's B operand.
    uint32_t b[kUnits][2][2][2];
    auto load_factor = [&](uint32_t kp, uint32_t group) {
        #pragma unroll
        for (uint32_t u = 0; u < kUnits; ++u) {
            #pragma unroll
            for (uint32_t s = 0; s < 2; ++s) {
                const uint32_t k = kp + (u * 8 + warp) * 32 + 16 * s + 4 * t;
                #pragma unroll
                for (uint32_t n = 0; n < 2; ++n) {
                    const uint32_t j = group * kGroupRanks + 8 * n + g;
                    float4 f = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (j < p.rank && k < k1) {
                        const float *src = static_cast<const float *>(p.a) + (k_major ? (size_t)k * p.rank + j : (size_t)j * p.K + k);
                        const size_t step = k_major ? p.rank : 1;
                        if (!k_major && p.a_vec) f = __ldg(reinterpret_cast<const float4 *>(src));
                        else f = make_float4(__ldg(src), __ldg(src + step), __ldg(src + 2 * step), __ldg(src + 3 * step));
                    }
                    const __half2 h0 = __floats2half2_rn(f.x, f.y), h1 = __floats2half2_rn(f.z, f.w);
                    b[u][s][n][0] = *reinterpret_cast<const uint32_t *>(&h0);
                    b[u][s][n][1] = *reinterpret_cast<const uint32_t *>(&h1);
                }
            }
        }
    };

    // ---- the rows' maxima (values that are not finite drop out) and factors ----
    uint32_t mx[4] = {};
    const uint32_t k_last = k0 + (max(k1, k0 + 1) - k0 - 1) / kPieceF32 * kPieceF32;  // the last part of the piece
    for (uint32_t kp = k0; kp <= k_last; kp += kPieceF32) {
        load(kp);
        if (kp == k_last) load_factor(kp, 0);
        #pragma unroll
        for (uint32_t u = 0; u < kUnits; ++u) {
            #pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                #pragma unroll
                for (uint32_t s = 0; s < 2; ++s) {
                    const uint32_t w[4] = {__float_as_uint(v[u][q][s].x), __float_as_uint(v[u][q][s].y), __float_as_uint(v[u][q][s].z), __float_as_uint(v[u][q][s].w)};
                    #pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if ((w[i] & 0x7fffffffu) < 0x7f800000u) mx[q] = max(mx[q], w[i] & 0x7fffffffu);
                }
            }
        }
    }
    const int w_exp = weight_exponent(p.absmax, p.scale_codes, p.scale_of_scales);
    #pragma unroll
    for (uint32_t q = 0; q < 4; ++q) {
        mx[q] = max(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], 1));
        mx[q] = max(mx[q], __shfl_xor_sync(0xffffffffu, mx[q], 2));
        if (t == 0) s_warp[warp][q * 8 + g] = mx[q];
    }
    __syncthreads();
    cluster.barrier_wait();
    {
        uint32_t m = 0;
        #pragma unroll
        for (uint32_t w = 0; w < 8; ++w) m = max(m, s_warp[w][lane]);
        for (uint32_t c = warp; c < cn; c += 8) cluster.map_shared_rank(&s_max[0][0], c)[rank_in * kRows + lane] = m;
    }
    cluster.sync();
    if (tid < kRows) {
        uint32_t m = 0;
        for (uint32_t c = 0; c < cn; ++c) m = max(m, s_max[c][tid]);
        const float sc = row_factor<true>(__uint_as_float(m));
        s_inv[tid] = 1.0f / sc;  // exact: sc is a power of two
        if (rank_in == 0 && m0 + tid < p.M) p.row_scale[m0 + tid] = sc * ldexpf(1.0f, w_exp);  // both factors of the outputs
    }
    __syncthreads();

    // ---- the products, and the copy ----
    // (The last piece's copy is written behind the arrival at the sums' exchange, whose release would wait for the stores.)
    uint32_t h[kUnits][4][2][2];
    auto copy = [&](uint32_t kp) {
        #pragma unroll
        for (uint32_t u = 0; u < kUnits; ++u) {
            const uint32_t k = kp + (u * 8 + warp) * 32 + 4 * t;
            #pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                const uint32_t m = m0 + q * 8 + g;
                #pragma unroll
                for (uint32_t s = 0; s < 2; ++s)
                    if (m < p.M && k < k1) *reinterpret_cast<uint2 *>(p.xh + (size_t)m * p.K + k + 16 * s) = make_uint2(h[u][q][s][0], h[u][q][s][1]);
            }
        }
    };
    uint32_t kp = k_last;  // (first, as its values are still there)
    for (;;) {
        #pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            const float is = s_inv[q * 8 + g];
            #pragma unroll
            for (uint32_t u = 0; u < kUnits; ++u) {
                #pragma unroll
                for (uint32_t s = 0; s < 2; ++s) {
                    const __half2 lo = __floats2half2_rn(v[u][q][s].x * is, v[u][q][s].y * is), hi = __floats2half2_rn(v[u][q][s].z * is, v[u][q][s].w * is);
                    h[u][q][s][0] = *reinterpret_cast<const uint32_t *>(&lo);
                    h[u][q][s][1] = *reinterpret_cast<const uint32_t *>(&hi);
                }
            }
        }
        for (uint32_t group = 0; group * kGroupRanks < p.rank; ++group) {
            if (group || kp != k_last) load_factor(kp, group);
            float acc[2][2][4] = {};  // of sixteen rows, of eight ranks
            #pragma unroll
            for (uint32_t u = 0; u < kUnits; ++u) {
                #pragma unroll
                for (uint32_t s = 0; s < 2; ++s) {
                    #pragma unroll
                    for (uint32_t q = 0; q < 2; ++q) {
                        #pragma unroll
                        for (uint32_t n = 0; n < 2; ++n)
                            ptx::mma_16816_f16(acc[q][n], h[u][2 * q][s][0], h[u][2 * q + 1][s][0], h[u][2 * q][s][1], h[u][2 * q + 1][s][1],
                                               b[u][s][n][0], b[u][s][n][1]);
                    }
                }
            }
            #pragma unroll
            for (uint32_t q = 0; q < 2; ++q) {
                #pragma unroll
                for (uint32_t n = 0; n < 2; ++n) {
                    *reinterpret_cast<float2 *>(&s_part[warp][q * 16 + g][8 * n + 2 * t]) = make_float2(acc[q][n][0], acc[q][n][1]);
                    *reinterpret_cast<float2 *>(&s_part[warp][q * 16 + 8 + g][8 * n + 2 * t]) = make_float2(acc[q][n][2], acc[q][n][3]);
                }
            }
            __syncthreads();
            {
                const uint32_t r = tid >> 3, c = (tid & 7u) * 2;
                float2 *const to = reinterpret_cast<float2 *>(&s_sum[r][group * kGroupRanks + c]);
                float2 sum = kp == k_last ? make_float2(0.0f, 0.0f) : *to;
                #pragma unroll
                for (uint32_t w = 0; w < 8; ++w) {  // in order
                    const float2 o = *reinterpret_cast<const float2 *>(&s_part[w][r][c]);
                    sum.x += o.x;
                    sum.y += o.y;
                }
                *to = sum;
            }
            __syncthreads();
        }
        const uint32_t next = kp == k_last ? k0 : kp + kPieceF32;
        if (next == k_last) break;
        copy(kp);
        kp = next;
        load(kp);
    }
    if (!p.rank) {
        copy(kp);
        return;
    }

    // ---- the CTAs' sums, each CTA a share of the rows; columns the adapter does not have are zeros ----
    // A row's sums go to the CTA whose share it is in, so that one meeting does: behind it nobody touches another CTA's memory.  (The
    // sums read from where they are, with a second meeting before a CTA leaves: 512 x 4096 x 4096 at rank 16 33.6 us instead of 32.8, 200 x
    // 8192 x 1024 at rank 64 33.7 instead of 32.1.)
    const uint32_t per = kRows / cn, rank_quads = p.rank / 4;  // (the rank is a multiple of four)
    for (uint32_t i = tid; i < kRows * rank_quads; i += kThreads) {
        const uint32_t r = i / rank_quads, c = i % rank_quads * 4;
        float *const to = cluster.map_shared_rank(s_all, r / per) + (rank_in * per + r % per) * kSumRow + c;
        *reinterpret_cast<float4 *>(to) = *reinterpret_cast<const float4 *>(&s_sum[r][c]);
    }
    __syncwarp();  // (lanes come from loops of different length)
    cluster.barrier_arrive();
    copy(kp);
    __syncwarp();
    cluster.barrier_wait();
    const float w_down = ldexpf(1.0f, -w_exp);
    const uint32_t quads = 16 * p.chunks, ld = 2 * 64 * p.chunks;
    for (uint32_t i = tid; i < per * quads; i += kThreads) {
        const uint32_t r = i / quads, c = i % quads * 4, m = m0 + rank_in * per + r;
        if (m >= p.M || (c >= p.rank && c < 2 * p.rank)) continue;
        float sum[4] = {};
        if (c < p.rank) {
            #pragma unroll 4
            for (uint32_t q = 0; q < cn; ++q) {
                const float4 w = *reinterpret_cast<const float4 *>(s_all + (q * per + r) * kSumRow + c);
                sum[0] += w.x;
                sum[1] += w.y;
                sum[2] += w.z;
                sum[3] += w.w;
            }
        }
        // (the products were taken with the scaled rows)
        put_halves(p.t_out, sum, p.scale * w_down, (size_t)m * ld + c, 64 * p.chunks);
        if (c < p.rank) put_halves(p.t_out, sum, p.scale * w_down, (size_t)m * ld + p.rank + c, 64 * p.chunks);
    }
}

// ---- the same for bf16 x and a factor on tcgen05: up to 64 ranks, rows of 16-byte pieces -------------------------------
// A cluster takes kRows (128, 64 or 32) rows of x, each CTA a piece of K in stages of 64 k.  One thread asks for a stage
// of x and of the factor by TMA (128-byte swizzle, a ring of eight stages), another issues its four MMAs (x the A
// operand as it lies, 128 rows whatever kRows is: the rows behind the tile are somebody else's bytes and nobody reads
// what they give; the factor the B operand, K-major as [r][K], MN-major as [K][r]), eight warps write the f16 copy and
// keep the maxima.  Nothing in the loop waits for the whole CTA: the kernel above, with warp MMAs, a barrier a stage
// and two stages in flight, ran at a fifth of the DRAM rate ([2048, 14336] at rank 64: 48 us, now 27).
constexpr uint32_t kTcThreads = 384, kTcStages = 8, kTcFactorStage = 8192;
__host__ __device__ constexpr uint32_t tc_ring(uint32_t rows) { return kTcStages * (rows * 128 + kTcFactorStage); }

template <int MODE, uint32_t kRows, bool k_major>
__global__ void __launch_bounds__(kTcThreads, 1)
prepass_tc_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_a, const Params p, const FailureRef failure) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    constexpr uint32_t kStages = kTcStages, kXStage = kRows * 128;
    // Eight warps convert: one a stage, two where it has 128 rows; a lane eight k of every fourth row.  A warp has the same
    // place of the ring every time (or two): it waits for all the place's rounds, so that a parity names the round.
    constexpr uint32_t kPerStage = kRows == 128 ? 2 : 1, kGroups = 8 / kPerStage, kWarpRows = kRows / kPerStage, kQuads = kWarpRows / 4;
    static_assert(kStages % kGroups == 0, "a warp's stages keep their places");
    constexpr bool kCopy = MODE == 0;
    static_assert(kRows * kPartPitch * 4 <= tc_ring(kRows), "the sums reuse the stages");
    static_assert((kStages - 1) * kXStage + 128 * 128 <= tc_ring(kRows), "an MMA reads 128 rows from the last stage's place");
    extern __shared__ uint8_t smem_any[];
    __shared__ uint32_t s_seen[kMaxCluster][kRows];  // the CTAs' rows (see row_seen)
    __shared__ uint32_t s_part[kGroups][kRows];      // this CTA's, by the warps
    __shared__ float s_inv[kRows];
    __shared__ float s_shift;
    __shared__ int s_exp;
    __shared__ __align__(8) uint64_t s_bars[2 * kStages + 1];
    __shared__ uint32_t s_tmem;
    uint8_t *const smem = smem_any + (1024u - (ptx::smem_addr(smem_any) & 1023u)) % 1024u;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t cn = cluster.num_blocks(), rank_in = cluster.block_rank();
    const uint32_t m0 = (blockIdx.x / cn) * kRows, k0 = min(rank_in * p.piece, p.K), k1 = min(k0 + p.piece, p.K);
    const uint32_t stages = (k1 - k0 + 63) / 64, base = ptx::smem_addr(smem), factor0 = base + kStages * kXStage;
    const uint32_t full0 = ptx::smem_addr(s_bars), empty0 = full0 + 8 * kStages, acc_bar = empty0 + 8 * kStages;
    float *part = reinterpret_cast<float *>(smem);
    const uint32_t n16 = (p.rank + 15) / 16 * 16;

    cluster.barrier_arrive();      // (waited for before the first access to another CTA's shared memory)
    auto request = [&](uint32_t st) {
        const uint32_t s = st % kStages, full = full0 + 8 * s;
        const int32_t k = (int32_t)(k0 + st * 64);
        ptx::mbar_arrive_expect_tx(full, kXStage + (k_major ? kTcFactorStage : n16 * 128));
        ptx::tma_load_2d(base + s * kXStage, &tmap_x, k, (int32_t)m0, full);
        ptx::tma_load_2d(factor0 + s * kTcFactorStage, &tmap_a, k_major ? 0 : k, k_major ? k : 0, full);
    };
    if (tid == 256) {  // (its loads are on their way while the others set up)
        for (uint32_t s = 0; s < kStages; ++s) {
            ptx::mbar_init(full0 + 8 * s, 1);
            ptx::mbar_init(empty0 + 8 * s, (kCopy ? kPerStage : 0) + 1);
        }
        ptx::mbar_init(acc_bar, 1);
        ptx::fence_mbar_init();
        ptx::fence_proxy_async();
        ptx::prefetch_tmap(&tmap_x);
        ptx::prefetch_tmap(&tmap_a);
        ptx::pdl_wait();
        for (uint32_t st = 0; st < min(stages, kStages); ++st) request(st);
    }
    if (warp == 9) {
        ptx::tmem_alloc(ptx::smem_addr(&s_tmem), 64);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();  // (what for: see the kernel above)
    if (blockIdx.x == 0)
        for (uint32_t i = tid; i < p.n_flags; i += kTcThreads) p.flags[i] = 0;
    const uint32_t acc = s_tmem;
    bool ok = true;
    if (warp == 11) {
        const int e = kCopy ? weight_exponent(p.absmax, p.scale_codes, p.scale_of_scales) : 0;
        if (lane == 0) s_exp = e;
    }
    if (kCopy && warp == 10) {
        // x comes over times a power of two that brings the largest of its first 256 values to [512, 1024): rows up to 32
        // times as large stay below 32768, and what is not exact in f16 then lies 2^-26 below those values, so that hardly
        // a row of ordinary values or of gradients needs to be written a second time (see below).
        uint32_t w = 0;
        if (lane * 8 < p.K) {
            const uint4 v = __ldg(static_cast<const uint4 *>(p.x) + lane);
            w = bf16x2_absmax(v.x, bf16x2_absmax(v.y, bf16x2_absmax(v.z, bf16x2_absmax(v.w, 0))));
        }
        const uint32_t m = __reduce_max_sync(0xffffffffu, bf16x2_larger_bits(w)), e = m >> 23;  // 136: [512, 1024)
        if (lane == 0) s_shift = e > 35 && e < 228 ? __uint_as_float((263 - e) << 23) : 1.0f;
    }
    if (kCopy && (warp == 10 || warp < 8)) asm volatile("bar.sync 1, 288;" ::: "memory");

    if (warp == 8) {
        if (lane == 0) {
            for (uint32_t st = kStages; st < stages; ++st) {
                if (!ptx::mbar_wait_suspended(empty0 + 8 * (st % kStages), (st / kStages + 1) & 1u)) {
                    ok = false;
                    break;
                }
                request(st);
            }
            if (!ok) NF4_REPORT_FAILURE(*failure.flag, *failure.host, 8);
        }
    } else if (warp == 9) {
        const uint32_t idesc = ptx::f16_idesc(1, 128, n16, false, k_major);
        for (uint32_t st = 0; st < stages; ++st) {
            const uint32_t s = st % kStages;
            ok = ptx::mbar_wait_suspended(full0 + 8 * s, (st / kStages) & 1u);
            if (!ok) break;
            ptx::tc_fence_after();
            if (ptx::elect_one()) {
                const uint64_t a = ptx::sw128_desc(base + s * kXStage), b = ptx::sw128_desc(factor0 + s * kTcFactorStage);
                #pragma unroll
                for (uint32_t i = 0; i < 4; ++i)  // 16 k: 32 bytes of a row, or sixteen rows
                    ptx::mma_ss_f16(acc, a + 2 * i, b + (k_major ? 128 : 2) * i, idesc, (st | i) != 0);
                ptx::tc_commit(empty0 + 8 * s);
                if (st + 1 == stages) ptx::tc_commit(acc_bar);
            }
            __syncwarp();
        }
        if (!ok && lane == 0) NF4_REPORT_FAILURE(*failure.flag, *failure.host, 9);
    } else if (kCopy && warp < 8) {
        // Every warp has stages of its own: a stage is read, converted and written in one go of many loads, and the next
        // ones are other warps' (eight warps to a stage waited for each link of its chain in turn: 30 us without the stores).
        const uint32_t piece = lane & 7u, r0 = warp % kPerStage * kWarpRows + (lane >> 3);
        uint32_t mx[kQuads] = {}, mn[kQuads];
        #pragma unroll
        for (uint32_t q = 0; q < kQuads; ++q) mn[q] = ~0u;
        const float shift = s_shift;
        for (uint32_t st = warp / kPerStage; st < stages; st += kGroups) {
            const uint32_t s = st % kStages;
            if (!ptx::mbar_wait_suspended(full0 + 8 * s, (st / kStages) & 1u)) {
                ok = false;
                break;
            }
            const uint32_t k = k0 + st * 64 + piece * 8, rows = k < k1 ? p.M - min(m0 + r0, p.M) : 0u;  // (from r0 on)
            __half *out = p.xh + (size_t)(m0 + r0) * p.K + k;
            constexpr uint32_t kBatch = 8;
            #pragma unroll
            for (uint32_t q0 = 0; q0 < kQuads; q0 += kBatch) {
                uint4 v[kBatch];
                #pragma unroll
                for (uint32_t q = 0; q < kBatch; ++q) {
                    const uint32_t r = r0 + (q0 + q) * 4;
                    v[q] = *reinterpret_cast<const uint4 *>(smem + s * kXStage + r * 128 + ((piece ^ (r & 7u)) << 4));
                }
                #pragma unroll
                for (uint32_t q = 0; q < kBatch; ++q, out += (size_t)4 * p.K) {
                    const uint32_t w[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
                    #pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        mx[q0 + q] = bf16x2_absmax(w[i], mx[q0 + q]);
                        mn[q0 + q] = bf16x2_absmin(w[i], mn[q0 + q]);
                    }
                    if ((q0 + q) * 4 < rows) *reinterpret_cast<uint4 *>(out) = bf16x8_to_f16x8(v[q], shift);
                }
            }
            __syncwarp();
            if (lane == 0) ptx::mbar_arrive(empty0 + 8 * s);
        }
        #pragma unroll
        for (uint32_t q = 0; q < kQuads; ++q) {  // (eight lanes hold a row's)
            uint32_t seen = row_seen(mx[q], mn[q]);
            #pragma unroll
            for (int d = 1; d < 8; d *= 2) seen = join_seen(seen, __shfl_xor_sync(0xffffffffu, seen, d));
            if (piece == 0) s_part[warp / kPerStage][r0 + q * 4] = seen;
        }
        if (!ok && lane == 0) NF4_REPORT_FAILURE(*failure.flag, *failure.host, 10);
    }
    if (!ok) ptx::let_flights_land();
    __syncwarp();
    __syncthreads();

    // The exchange.  Only the last four warps, which have written nothing to global memory, release what they do here: a
    // release by the others would wait for the copy's stores.
    if (warp >= 8 && warp - 8 < kRows / 32) {
        // this CTA's sums, a lane a row; columns the factor does not have are zeros
        const uint32_t q = warp - 8;
        if (stages && !ptx::mbar_wait_suspended(acc_bar, 0)) {
            if (lane == 0) NF4_REPORT_FAILURE(*failure.flag, *failure.host, 11);
        }
        ptx::tc_fence_after();
        #pragma unroll
        for (uint32_t c = 0; c < 64; c += 16) {
            uint32_t v[16];
            ptx::tmem_ld16(acc + ((q * 32) << 16) + c, v);
            ptx::tmem_wait_ld();
            const bool real = c < n16 && stages;
            float4 *dst = reinterpret_cast<float4 *>(part + (q * 32 + lane) * kPartPitch + c);
            #pragma unroll
            for (int i = 0; i < 4; ++i)
                dst[i] = real ? make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]), __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]))
                              : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        ptx::tc_fence_before();
    }
    cluster.barrier_wait();
    if (kCopy && warp >= 8) {
        const uint32_t r = (tid - 256) % kRows;
        uint32_t seen = s_part[0][r];
        #pragma unroll
        for (uint32_t g = 1; g < kGroups; ++g) seen = join_seen(seen, s_part[g][r]);
        for (uint32_t c = (tid - 256) / kRows; c < cn; c += 128 / kRows) cluster.map_shared_rank(&s_seen[0][0], c)[rank_in * kRows + r] = seen;
    }
    if (warp >= 8) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    else asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    const int w_exp = s_exp;
    if (kCopy) {
        if (tid < kRows) {
            uint32_t seen = s_seen[0][tid];
            for (uint32_t c = 1; c < cn; ++c) seen = join_seen(seen, s_seen[c][tid]);
            // A row's own factor brings its largest value to [16384, 32768); one with an infinity has none.  The copy is
            // left as it is where it holds every value exactly: nothing too large, and nothing below 2^-17 (eight bits
            // down to f16's last, 2^-24).  The row's own copy is then exact as well, so that what the GEMM sees of a row
            // does not depend on the values the common factor came from.
            const float mx = __uint_as_float(seen & 0xffff0000u), least = __uint_as_float((seen & 0x7fffu) << 16);
            const bool exact = mx * s_shift <= 32768.0f && least * s_shift >= 7.62939453125e-6f;
            const float sc = exact ? 1.0f / s_shift : mx < __int_as_float(0x7f800000) ? row_factor<true>(mx) : 1.0f;
            s_inv[tid] = 1.0f / sc;  // exact: sc is a power of two
            if (rank_in == 0 && m0 + tid < p.M) p.row_scale[m0 + tid] = sc * ldexpf(1.0f, w_exp);  // both factors of the outputs
        }
        __syncthreads();
        for (uint32_t r = warp; r < kRows; r += kTcThreads / 32) {  // the rare rows with a factor of their own, again
            const float is = s_inv[r];
            if (is == s_shift || m0 + r >= p.M) continue;
            for (uint32_t k = k0 + lane * 8; k < k1; k += 256) {
                const size_t at = (size_t)(m0 + r) * p.K + k;
                *reinterpret_cast<uint4 *>(p.xh + at) = bf16x8_to_f16x8(__ldg(reinterpret_cast<const uint4 *>(static_cast<const uint16_t *>(p.x) + at)), is);
            }
        }
    }
    const float w_down = ldexpf(1.0f, -w_exp);
    const uint32_t per = (kRows + cn - 1) / cn;  // rows of this CTA's share
    for (uint32_t i = tid; i < per * 16; i += kTcThreads) {
        const uint32_t r = rank_in * per + (i >> 4), c = (i & 15u) * 4, m = m0 + r;
        if (r >= kRows || m >= p.M) continue;
        float sum[4] = {};
        #pragma unroll 4
        for (uint32_t q = 0; q < cn; ++q) {
            const float4 w = *reinterpret_cast<const float4 *>(cluster.map_shared_rank(part, q) + r * kPartPitch + c);
            sum[0] += w.x;
            sum[1] += w.y;
            sum[2] += w.z;
            sum[3] += w.w;
        }
        put_halves(kCopy ? p.t_out : nullptr, sum, p.scale * (kCopy ? s_inv[r] : 1.0f) * w_down, (size_t)m * 128 + c, 64);
        put_halves(p.r_out, sum, 1.0f, (size_t)m * 128 + c, 64);
    }
    ptx::tc_fence_before();
    __syncwarp();  // (lanes come from loops of different length)
    ptx::cluster_sync_all();  // the sums have been read, before a CTA leaves (a relaxed arrival would not say so)
    if (warp == 9) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(acc, 64);
    }
}

}  // namespace

namespace {

template <uint32_t kRows>
auto tc_kernel(bool copy, bool k_major) {
    return copy ? (k_major ? prepass_tc_kernel<0, kRows, true> : prepass_tc_kernel<0, kRows, false>)
                : (k_major ? prepass_tc_kernel<2, kRows, true> : prepass_tc_kernel<2, kRows, false>);
}

int32_t launch_tc(const PrepassArgs &q, Params &p, cudaStream_t stream) {
    // Rows to a cluster: what leaves an SM the least to fetch, its stages of x and the factor (an SM holds one CTA).
    uint32_t rows = 0, cn = 1;
    uint64_t least = 0;
    decltype(tc_kernel<128>(true, true)) kernel = nullptr;
    for (uint32_t r : {128u, 64u, 32u}) {
        const bool copy = q.xh != nullptr;
        auto k = r == 128 ? tc_kernel<128>(copy, q.k_major) : r == 64 ? tc_kernel<64>(copy, q.k_major) : tc_kernel<32>(copy, q.k_major);
        ClusterRoom room;
        NF4_TRY(cluster_room(reinterpret_cast<const void *>(k), kTcThreads, tc_ring(r) + 1024, &room));
        const uint64_t tiles = (q.M + r - 1) / r;
        for (uint32_t c = 1; c <= kMaxCluster && (c == 1 || (tiles <= room.any[c] && q.K > 64ull * (c - 1))); ++c) {
            const uint64_t stages = (q.K + 64ull * c - 1) / (64ull * c), waves = (tiles * c + kNumSMs - 1) / kNumSMs;
            const uint64_t cost = waves * stages * (r * 128 + kTcFactorStage);
            if (kernel && cost >= least) continue;
            least = cost;
            rows = r;
            cn = c;
            kernel = k;
        }
    }
    const uint64_t tiles = (q.M + rows - 1) / rows;
    if (tiles * cn >= (1ull << 31)) return fail(NF4_ERR_UNSUPPORTED, "activations_prepass: too many rows");
    p.piece = ((q.K + cn - 1) / cn + 63) / 64 * 64;
    CUtensorMap map_x, map_a;
    NF4_TRY(make_map(&map_x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, q.x, q.M, q.K, (uint64_t)q.K * 2, rows, 64, CU_TENSOR_MAP_SWIZZLE_128B));
    if (q.k_major)
        NF4_TRY(make_map(&map_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, q.a, q.K, q.rank, (uint64_t)q.rank * 2, 64, 64, CU_TENSOR_MAP_SWIZZLE_128B));
    else
        NF4_TRY(make_map(&map_a, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, q.a, q.rank, q.K, (uint64_t)q.K * 2, (q.rank + 15) / 16 * 16, 64,
                         CU_TENSOR_MAP_SWIZZLE_128B));
    FailureRef failure;
    NF4_TRY(prefill_failure_ref(&failure));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(tiles * cn));
    cfg.blockDim = dim3(kTcThreads);
    cfg.dynamicSmemBytes = tc_ring(rows) + 1024;
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
    return check_cuda(cudaLaunchKernelEx(&cfg, kernel, map_x, map_a, p, failure), "prepass_tc_kernel launch");
}

}  // namespace

int32_t activations_prepass(const PrepassArgs &q, cudaStream_t stream) {
    if (q.x_f32 && (!q.xh || q.r_out || q.rank > kMostRanks || q.rank % 4))
        return fail(NF4_ERR_UNSUPPORTED, "activations_prepass: f32 with the copy, without r_out, and at most %u ranks", kMostRanks);
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
    p.chunks = ((q.x_f32 ? 2 * q.rank : q.rank) + 63) / 64;
    p.a_vec = aligned16(q.a) && (q.k_major ? q.rank : q.K) % 8 == 0;
    p.scale = q.scale;
    // The tcgen05 kernel, where its TMA takes the tensors: always for the product alone ([16, 11008] and [14, 768] the same
    // time); with the copy from four million values on (whole forwards to 512 columns: [1024, 4096] at rank 64 42.7 -> 40.3 us,
    // [4096, 1024] 23.7 -> 23.1, but [512, 2048] 27.5 -> 30.3 and [256, 4096] at rank 16 the other way too: an SM
    // holds one of its CTAs and two of the other's), and never without a factor ([2048, 4096]: 39.2 -> 41.1).
    const bool tc_shape = !q.x_f32 && q.rank && q.rank <= 64 && q.K % 8 == 0 && aligned16(q.x) && p.a_vec;
    if (tc_shape && (!q.xh || (uint64_t)q.M * q.K >= 1u << 22)) return launch_tc(q, p, stream);
    // 64 rows to a cluster beyond 512 rows, where the clusters of 32 no longer fit the chip at once, else 32 (half of the
    // factor's traffic against more CTAs)
    const uint32_t rows = !q.x_f32 && q.M > 512 ? 64 : 32;
    const uint64_t tiles = (q.M + rows - 1) / rows;
    auto pick = [&](auto km) {
        constexpr bool k_major = decltype(km)::value;
        if (q.x_f32) return prepass_f32_kernel<k_major>;
        return rows == 64 ? (q.xh ? prepass_kernel<0, 64, k_major> : prepass_kernel<2, 64, k_major>)
                          : (q.xh ? prepass_kernel<0, 32, k_major> : prepass_kernel<2, 32, k_major>);
    };
    auto kernel = q.k_major ? pick(std::true_type{}) : pick(std::false_type{});
    const int smem = (int)(q.x_f32 ? rows * kSumRow * sizeof(float) : stages_of(rows) * stage_bytes(rows));
    // as many CTAs of K as the chip holds at once, two on an SM (a second wave took 21 us where one takes 11; of f32 [4096, 4096]
    // two CTAs to a cluster 40 us, eight, whose pieces are read once, 45; [4096, 14336] 121 and, sixteen, 154)
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
