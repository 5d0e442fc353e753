// What the tensor-core GEMM needs of the activations before it runs, and the adapter intermediate for
// the gradients: in one pass over x [M][K]
//   xh[m][k] = f16(x[m][k] / row_scale[m])  (row_scale: a power of two),
//   T = scale (x A^T) / row_scale as bf16 hi / lo halves (more k-steps of the GEMM),
//   R = x A^T likewise, unscaled (the operand of the gradient kernel).
//
// Split.  A cluster of CTAs takes 32 rows of x, each CTA a piece of K, which it brings into shared
// memory once (16-byte asynchronous copies): the row maxima, the conversion and the products all read it
// there.  The CTAs' maxima and partial sums of T meet through distributed shared memory, in rank order
// (results do not depend on timing).  The adapter factor streams through shared memory in stages of 64
// k in whichever orientation it is stored: [r][K] is the MMA's B operand as it lies, [K][r] through
// transposing matrix loads.  Bound by the bytes of x in and xh out; before, a CTA took 16 rows over the
// whole of K and read all of A for them (20 us for x [2048, 4096] at rank 64, 64 for K = 14336; few rows
// left most SMs idle: 14 us for 203 rows).
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "kernels.cuh"
#include "ptx.cuh"

namespace nf4 {
namespace {

constexpr uint32_t kRows = 32, kThreads = 256, kStageK = 64, kStages = 3;
constexpr uint32_t kFactorPitch = 144, kFactorStage = 64 * kFactorPitch;  // 64 rows of 128 bytes, 16 of padding
constexpr uint32_t kPartPitch = 68;                                        // floats
constexpr uint32_t kMaxCluster = 16;
static_assert(kRows * kPartPitch * 4 <= kStages * kFactorStage, "the sums reuse the factor's stages");

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
    uint32_t M, K, rank, chunks, k_major;
    uint32_t a_vec;        // the factor's rows are 16-byte aligned
    uint32_t piece, sub;   // k per CTA; k of it in shared memory at a time (the whole piece unless K is huge): multiples of 64
    float scale;
    uint32_t wait_late;    // see activations_prepass
};

// Running maxima of |bf16|, a pair at a time; a NaN leaves the maximum as it is (max.bf16x2
// returns the other operand).
__device__ __forceinline__ uint32_t bf16x2_absmax(uint32_t w, uint32_t mx) {
    uint32_t d;
    asm("max.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(w & 0x7fff7fffu), "r"(mx));
    return d;
}
// The larger half of such a pair as an f32 pattern; 0 if only NaNs were seen.
__device__ __forceinline__ uint32_t bf16x2_larger_bits(uint32_t mx) {
    const uint32_t lo = mx << 16, hi = mx & 0xffff0000u;
    const uint32_t a = lo <= 0x7f800000u ? lo : 0u, b = hi <= 0x7f800000u ? hi : 0u;
    return max(a, b);
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
template <int MODE>
__global__ void __launch_bounds__(kThreads)
prepass_kernel(const Params p) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    constexpr bool F32 = MODE == 1;
    constexpr uint32_t kElem = F32 ? 4 : 2;
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint32_t s_max[kMaxCluster][kRows];   // the CTAs' row maxima (f32 patterns)
    __shared__ float s_inv[kRows];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t cn = cluster.num_blocks(), rank_in = cluster.block_rank();
    const uint32_t m0 = (blockIdx.x / cn) * kRows, k0 = min(rank_in * p.piece, p.K), k1 = min(k0 + p.piece, p.K);
    const uint32_t nst = (k1 - k0 + kStageK - 1) / kStageK;          // stages of 64 k of this CTA
    const uint32_t sub_stages = p.sub / kStageK, subs = (nst + sub_stages - 1) / sub_stages;
    const bool resident = subs <= 1;
    const uint32_t pitch = p.sub * kElem + 16;       // 16 mod 128: matrix loads hit all banks
    uint8_t *stages = smem + kRows * pitch;
    const uint32_t xt = ptx::smem_addr(smem), ft = ptx::smem_addr(stages);
    float *part = reinterpret_cast<float *>(stages);

    cluster.barrier_arrive();      // (waited for before the first access to another CTA's shared memory)
    // the GEMM may set itself up and start on the weights, which are in place once the kernels before this
    // one have completed (a repacked weight it waits for itself)
    if (!p.wait_late) ptx::pdl_wait();
    ptx::pdl_launch_dependents();
    // the GEMM's CTAs raise these once this kernel has completed (their readers and writers wait for that)
    if (blockIdx.x == 0)
        for (uint32_t i = tid; i < p.n_flags; i += kThreads) p.flags[i] = 0;

    // x's k of stages [s0, s1) into shared memory; missing rows and the ragged end of K as zeros
    auto load_x = [&](uint32_t s0, uint32_t s1) {
        const uint32_t pieces = (s1 - s0) * kStageK * kElem / 16;  // per row
        for (uint32_t i = tid; i < kRows * pieces; i += kThreads) {
            const uint32_t r = i / pieces, c = i - r * pieces, k = k0 + s0 * kStageK + c * (16 / kElem);
            const bool real = m0 + r < p.M && k < k1;
            ptx::cp_async_16_or_zero(xt + r * pitch + c * 16,
                                     static_cast<const uint8_t *>(p.x) + (real ? ((size_t)(m0 + r) * p.K + k) * kElem : 0), real);
        }
        ptx::cp_async_commit();
    };
    const uint16_t *a = static_cast<const uint16_t *>(p.a);
    auto load_factor = [&](uint32_t st, uint32_t chunk) {  // stage st of the factor's 64 ranks `chunk`
        if (st < nst) {
            const uint32_t dst = ft + (st % kStages) * kFactorStage, ks = k0 + st * kStageK, j0 = chunk * 64;
            if (!p.a_vec) {  // rows at odd places: element by element
                for (uint32_t i = tid; i < 64 * 64; i += kThreads) {
                    const uint32_t r = i >> 6, c = i & 63u, k = ks + (p.k_major ? r : c), j = j0 + (p.k_major ? c : r);
                    const uint16_t v = k < k1 && j < p.rank ? __ldg(a + (p.k_major ? (size_t)k * p.rank + j : (size_t)j * p.K + k)) : (uint16_t)0;
                    *reinterpret_cast<uint16_t *>(stages + (st % kStages) * kFactorStage + r * kFactorPitch + c * 2) = v;
                }
            } else {
                #pragma unroll
                for (uint32_t q = 0; q < 2; ++q) {
                    const uint32_t i = tid + q * kThreads, r = i >> 3, c = i & 7u;
                    // row r of the stage: rank j0 + r, or k = ks + r
                    const bool real = p.k_major ? ks + r < k1 && j0 + c * 8 < p.rank : j0 + r < p.rank && ks + c * 8 < k1;
                    const size_t at = p.k_major ? (size_t)(ks + r) * p.rank + j0 + c * 8 : (size_t)(j0 + r) * p.K + ks + c * 8;
                    ptx::cp_async_16_or_zero(dst + r * kFactorPitch + c * 16, a + (real ? at : 0), real);
                }
            }
        }
        ptx::cp_async_commit();
    };
    if (resident) load_x(0, nst);
    if (p.rank) {
        load_factor(0, 0);
        load_factor(1, 0);
    }

    // ---- row maxima; a warp has four rows ----
    if (MODE != 2) {
        uint32_t mx[4] = {0, 0, 0, 0};
        for (uint32_t s = 0; s < subs; ++s) {
            const uint32_t s0 = s * sub_stages, s1 = min(nst, s0 + sub_stages);
            if (!resident) {
                __syncthreads();
                load_x(s0, s1);
                ptx::cp_async_wait<0>();
            } else if (p.rank) {
                ptx::cp_async_wait<2>();
            } else {
                ptx::cp_async_wait<0>();
            }
            __syncthreads();
            #pragma unroll
            for (uint32_t q = 0; q < 4; ++q) {
                const uint4 *row = reinterpret_cast<const uint4 *>(smem + (warp * 4 + q) * pitch);
                for (uint32_t c = lane; c < (s1 - s0) * kStageK * kElem / 16; c += 32) {
                    const uint4 v = row[c];
                    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
                    #pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (F32) {
                            const uint32_t b = w[i] & 0x7fffffffu;
                            if (b < 0x7f800000u) mx[q] = max(mx[q], b);
                        } else {
                            mx[q] = bf16x2_absmax(w[i], mx[q]);
                        }
                    }
                }
            }
        }
        cluster.barrier_wait();
        #pragma unroll
        for (uint32_t q = 0; q < 4; ++q) {
            const uint32_t m = __reduce_max_sync(0xffffffffu, F32 ? mx[q] : bf16x2_larger_bits(mx[q]));
            if (lane < cn) cluster.map_shared_rank(&s_max[0][0], lane)[rank_in * kRows + warp * 4 + q] = m;  // to every CTA
        }
        cluster.sync();
        const int w_exp = weight_exponent(p.absmax, p.scale_codes, p.scale_of_scales);
        if (tid < kRows) {
            uint32_t m = 0;
            for (uint32_t c = 0; c < cn; ++c) m = max(m, s_max[c][tid]);
            const float sc = row_factor<F32>(__uint_as_float(m));
            s_inv[tid] = 1.0f / sc;  // exact: sc is a power of two
            if (rank_in == 0 && m0 + tid < p.M) p.row_scale[m0 + tid] = sc * ldexpf(1.0f, w_exp);  // both factors of the outputs
        }
        __syncthreads();
    } else {
        cluster.barrier_wait();
    }

    // The f16 copy of stages [s0, s1) (MODE 1: also in place, for the products), a warp four rows.
    auto convert = [&](uint32_t s0, uint32_t s1, bool store) {
        #pragma unroll 1
        for (uint32_t q = 0; q < 4; ++q) {
            const uint32_t r = warp * 4 + q, n8 = (s1 - s0) * kStageK / 8;
            const float is = s_inv[r];
            uint8_t *row = smem + r * pitch;
            const uint32_t ks = k0 + s0 * kStageK;
            uint4 *out = reinterpret_cast<uint4 *>(p.xh + (size_t)(m0 + r) * p.K + ks);
            const bool live = store && m0 + r < p.M;
            for (uint32_t c0 = 0; c0 < n8; c0 += 32) {  // eight values per lane
                const uint32_t c = c0 + lane;
                const bool in = c < n8;
                uint4 o = make_uint4(0, 0, 0, 0);
                if (F32) {
                    if (in) {
                        const float4 u = reinterpret_cast<const float4 *>(row)[2 * c], v = reinterpret_cast<const float4 *>(row)[2 * c + 1];
                        const __half2 h0 = __floats2half2_rn(u.x * is, u.y * is), h1 = __floats2half2_rn(u.z * is, u.w * is);
                        const __half2 h2 = __floats2half2_rn(v.x * is, v.y * is), h3 = __floats2half2_rn(v.z * is, v.w * is);
                        o = make_uint4(*reinterpret_cast<const uint32_t *>(&h0), *reinterpret_cast<const uint32_t *>(&h1),
                                       *reinterpret_cast<const uint32_t *>(&h2), *reinterpret_cast<const uint32_t *>(&h3));
                    }
                    __syncwarp();  // the f32 of these 32 lanes have been read; their f16 fill the first half of that place
                    if (in) reinterpret_cast<uint4 *>(row)[c] = o;
                    __syncwarp();
                } else if (in) {
                    o = bf16x8_to_f16x8(reinterpret_cast<const uint4 *>(row)[c], is);
                }
                if (live && in && ks + c * 8 < k1) out[c] = o;
            }
        }
    };

    // ---- the products: per stage of 64 k a warp has 16 rows and 16 k, 64 ranks at a time ----
    const uint32_t rh = warp & 1u, kq = warp >> 1, g = lane >> 2, t = lane & 3u, li = lane >> 3, lr = lane & 7u;
    const float w_down = MODE == 2 ? 1.0f : ldexpf(1.0f, -weight_exponent(p.absmax, p.scale_codes, p.scale_of_scales));
    for (uint32_t chunk = 0; chunk < max(p.chunks, 1u); ++chunk) {
        float acc[8][4];
        #pragma unroll
        for (int u = 0; u < 8; ++u) acc[u][0] = acc[u][1] = acc[u][2] = acc[u][3] = 0.0f;
        const uint32_t tiles16 = p.rank ? (min(64u, p.rank - chunk * 64) + 15) / 16 : 0u;
        if (chunk) {
            load_factor(0, chunk);
            load_factor(1, chunk);
        }
        const uint32_t a_at = xt + (rh * 16 + (li & 1u) * 8 + lr) * pitch + (kq * 16 + (li >> 1) * 8) * 2;
        const uint32_t b_at = p.k_major ? (kq * 16 + (li & 1u) * 8 + lr) * kFactorPitch + (li >> 1) * 16
                                        : ((li >> 1) * 8 + lr) * kFactorPitch + (kq * 16 + (li & 1u) * 8) * 2;
        for (uint32_t s = 0; s < subs; ++s) {
            const uint32_t s0 = s * sub_stages, s1 = min(nst, s0 + sub_stages);
            if (!resident) {
                __syncthreads();
                load_x(s0, s1);
                ptx::cp_async_wait<0>();
                __syncthreads();
            }
            if (MODE != 2 && (chunk == 0 || (F32 && !resident))) {
                convert(s0, s1, chunk == 0);
                if (F32) __syncthreads();
            }
            if (!p.rank) continue;
            for (uint32_t st = s0; st < s1; ++st) {
                ptx::cp_async_wait<1>();
                __syncthreads();
                load_factor(st + 2, chunk);
                uint32_t af[4];
                ptx::ldmatrix_x4(af, a_at + (st - s0) * (kStageK * 2));
                const uint32_t bs = ft + (st % kStages) * kFactorStage + b_at;
                #pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    if (u >= tiles16) break;
                    uint32_t bf[4];
                    if (p.k_major) ptx::ldmatrix_x4_trans(bf, bs + u * 32);
                    else ptx::ldmatrix_x4(bf, bs + u * 16 * kFactorPitch);
                    if (F32) {
                        ptx::mma_16816_f16(acc[2 * u], af[0], af[1], af[2], af[3], bf[0], bf[1]);
                        ptx::mma_16816_f16(acc[2 * u + 1], af[0], af[1], af[2], af[3], bf[2], bf[3]);
                    } else {
                        ptx::mma_16816_bf16(acc[2 * u], af[0], af[1], af[2], af[3], bf[0], bf[1]);
                        ptx::mma_16816_bf16(acc[2 * u + 1], af[0], af[1], af[2], af[3], bf[2], bf[3]);
                    }
                }
            }
        }
        if (!p.rank) break;
        ptx::cp_async_wait<0>();
        // the four k-quarters add up in turn, then the CTAs of the cluster in rank order
        for (uint32_t turn = 0; turn < 4; ++turn) {
            __syncthreads();
            if (kq == turn) {
                #pragma unroll
                for (int u = 0; u < 8; ++u) {
                    float2 *lo = reinterpret_cast<float2 *>(part + (rh * 16 + g) * kPartPitch + 8 * u + 2 * t);
                    float2 *hi = reinterpret_cast<float2 *>(part + (rh * 16 + g + 8) * kPartPitch + 8 * u + 2 * t);
                    const float2 l = turn ? *lo : make_float2(0.0f, 0.0f), h = turn ? *hi : make_float2(0.0f, 0.0f);
                    *lo = make_float2(l.x + acc[u][0], l.y + acc[u][1]);
                    *hi = make_float2(h.x + acc[u][2], h.y + acc[u][3]);
                }
            }
        }
        cluster.sync();
        const uint32_t per = kRows / cn, ld = 2 * 64 * p.chunks;
        for (uint32_t i = tid; i < per * 64; i += kThreads) {
            const uint32_t r = rank_in * per + (i >> 6), c = i & 63u, m = m0 + r;
            float sum = 0.0f;
            for (uint32_t q = 0; q < cn; ++q) sum += cluster.map_shared_rank(part, q)[r * kPartPitch + c];
            if (m < p.M) {
                const size_t at = (size_t)m * ld + chunk * 64 + c;
                if (MODE != 2) {
                    // (MODE 1: the products were taken with the scaled rows)
                    const float v = sum * p.scale * (F32 ? 1.0f : s_inv[r]) * w_down;
                    const __nv_bfloat16 hi = __float2bfloat16_rn(v);
                    p.t_out[at] = hi;
                    p.t_out[at + 64 * p.chunks] = __float2bfloat16_rn(v - __bfloat162float(hi));
                }
                if (MODE == 2 || p.r_out) {
                    const __nv_bfloat16 hi = __float2bfloat16_rn(sum);
                    p.r_out[at] = hi;
                    p.r_out[at + 64 * p.chunks] = __float2bfloat16_rn(sum - __bfloat162float(hi));
                }
            }
        }
        cluster.sync();  // the sums have been read (before the next chunk's stages, and before a CTA leaves)
    }
    if (p.wait_late) ptx::pdl_wait();
}

}  // namespace

int32_t activations_prepass(const PrepassArgs &q, cudaStream_t stream) {
    const uint32_t esize = q.x_f32 ? 4 : 2;
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
    p.k_major = q.k_major;
    p.a_vec = aligned16(q.a) && (q.k_major ? q.rank : q.K) % 8 == 0;
    p.scale = q.scale;
    p.wait_late = q.beside_predecessor;
    // CTAs per 32 rows: pieces of at most 512 k (x and the stages then leave room for three CTAs on an
    // SM), sixteen CTAs at most; shorter pieces where there are few rows, to have all SMs read
    const uint64_t tiles = (q.M + kRows - 1) / kRows;
    uint32_t cn = 1;
    while (cn < kMaxCluster && ((q.K + cn - 1) / cn > 512 || (tiles * cn < 148 && (q.K + cn - 1) / cn > 256))) cn *= 2;
    p.piece = ((q.K + cn - 1) / cn + kStageK - 1) / kStageK * kStageK;
    const uint32_t most = (224 * 1024 - kStages * kFactorStage) / kRows / esize / kStageK * kStageK - kStageK;
    p.sub = p.piece < most ? p.piece : most;
    const int smem = (int)(kRows * (p.sub * esize + 16) + kStages * kFactorStage);
    if (tiles * cn >= (1ull << 31)) return fail(NF4_ERR_UNSUPPORTED, "activations_prepass: too many rows");
    auto kernel = q.x_f32 ? prepass_kernel<1> : q.xh ? prepass_kernel<0> : prepass_kernel<2>;
    NF4_TRY(ensure_dynamic_smem(reinterpret_cast<const void *>(kernel), 224 * 1024));
    if (cn > 8) NF4_TRY(allow_large_clusters(reinterpret_cast<const void *>(kernel)));
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
