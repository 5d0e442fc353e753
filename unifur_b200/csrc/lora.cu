// The adapter by itself: LoraAdapter::forward, LoraAdapter::delta_weight and QLoraLinear::merged of
// the reference (src/quantize.rs:620-624, 629-634, 717-726), and the gather step of the
// column-sharded forward.  Small CUDA-core kernels: a rank-r product has r multiply-adds per
// output, so these are bound by the bytes of x, A, B and the output they touch.
//
// Arithmetic follows the reference's order in f32: (x A) first, then (.) B, the scale last;
// delta = (A B) * scale; merged = W + delta with W = level * block scale.
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <dlfcn.h>

#include <mutex>

#include "kernels.cuh"
#include "ptx.cuh"

namespace nf4 {
namespace {

template <class T>
__device__ __forceinline__ float to_f32(T v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

template <class T>
__device__ __forceinline__ T from_f32(float v);
template <>
__device__ __forceinline__ float from_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f32<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// A(k, j) and B(j, n) in either orientation:
//   OUT_IN: A [r, d_in], B [d_out, r]      IN_OUT (the reference's): A [d_in, r], B [r, d_out]
template <class T>
__device__ __forceinline__ float a_at(const T *a, int32_t layout, uint64_t k, uint64_t j, uint64_t d_in, uint32_t rank) {
    return to_f32<T>(layout == NF4_LAYOUT_OUT_IN ? a[j * d_in + k] : a[k * rank + j]);
}
template <class T>
__device__ __forceinline__ float b_at(const T *b, int32_t layout, uint64_t j, uint64_t n, uint64_t d_out, uint32_t rank) {
    return to_f32<T>(layout == NF4_LAYOUT_OUT_IN ? b[n * rank + j] : b[j * d_out + n]);
}

// Products with a thin side, in f32: out(i, j) = f sum_q L(q, i) R(q, j), j a rank.  The intermediates T = x A and U = grad_y B^T
// (i a row, q a column of x) and the adapter's gradients (i a column of X, q a row; R the other intermediate).
// A CTA takes 64 i and kJ ranks; q comes in stages of 32 through two places of shared memory, the next stage's values in
// registers while one is multiplied.  A thread has 4 x 4 outputs, so that two 16-byte loads feed sixteen multiply-adds; with
// fewer ranks than 64 the threads form groups that divide a stage's q.  The CTAs that share a tile's q form a cluster: their sums
// meet through distributed shared memory, in rank order.  Sums of 32 products are added to the sums so far, so that errors
// grow with the square root of Q / 32 and not of Q.
// Bound by the multiply-adds and, at few rows, by the bytes of the factors.  Two products (or two gradients) are one launch.
// One warp to an output, or one CTA to eight rows or 32 columns, before: 2048 x 4096 x 4096 in f32 at rank 64, T 67 us, U 206, the
// gradients 177 each; now 83 for T and U and 78 for both gradients.  512 x 4096 x 4096 at rank 16: 79, 20, 46 and 46; now 17 and 14.
// The relative error against 64 bits: 2.6e-7 to 8.6e-7 before, now 1.0e-7 to 2.2e-7 (seven sizes up to Q = 20480).
struct ThinJob {
    const void *l, *r;
    void *out;
    uint64_t I, Q, tiles;
    uint64_t share;        // q of a CTA of the cluster
    float f;
    uint32_t l_vec;        // L's rows are whole, aligned vectors of four
    uint32_t r_j_major;    // R(q, j) = r[j * Q + q], else r[q * rank + j]
    uint32_t out_j_major;  // out[j * I + i], else out[i * rank + j]
};
struct ThinParams {
    ThinJob job[2];
    uint32_t rank;
};
constexpr uint32_t kThinI = 64, kThinQ = 32, kThinPitch = kThinI + 4;

template <class T>
__device__ __forceinline__ float4 load_four(const T *p, bool vec, uint64_t n) {  // the first n of four, zeros behind
    if (vec && n >= 4) {
        if constexpr (sizeof(T) == 4) return __ldg(reinterpret_cast<const float4 *>(p));
        const uint2 v = __ldg(reinterpret_cast<const uint2 *>(p));
        return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
    }
    return make_float4(n > 0 ? to_f32<T>(p[0]) : 0.0f, n > 1 ? to_f32<T>(p[1]) : 0.0f, n > 2 ? to_f32<T>(p[2]) : 0.0f, n > 3 ? to_f32<T>(p[3]) : 0.0f);
}

// TL, TR, TO: types of L, R and the output.  kQMajor: L(q, i) = l[q * I + i], else l[i * Q + q].
template <class TL, class TR, class TO, bool kQMajor, uint32_t kJ>
__global__ void __launch_bounds__(256)
thin_product_kernel(const ThinParams p) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    constexpr uint32_t kTile = kThinI / 4 * (kJ / 4), kGroups = 256 / kTile, kOwn = kThinQ / kGroups, kRs = kJ + 4, kEach = kThinQ * kJ / 256;
    static_assert(kThinI * kRs * kGroups <= 2 * kThinQ * (kThinPitch + kRs), "the groups' sums reuse the stages");
    __shared__ __align__(16) float smem[2 * kThinQ * (kThinPitch + kRs)];
    __shared__ __align__(16) float s_apart[kGroups > 1 ? kThinI * kRs : 4];
    float *const s_sum = kGroups > 1 ? s_apart : smem;  // this CTA's sums [64][kRs]
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, cn = cluster.num_blocks(), rank_in = cluster.block_rank();
    const uint64_t all_tile = blockIdx.x / cn;
    const ThinJob &job = p.job[all_tile < p.job[0].tiles ? 0 : 1];
    const uint64_t i0 = (all_tile < p.job[0].tiles ? all_tile : all_tile - p.job[0].tiles) * kThinI;
    const uint64_t q0 = min(rank_in * job.share, job.Q), q1 = min(q0 + job.share, job.Q);
    const uint32_t j0 = blockIdx.y * kJ;
    // A thread's two vectors of L of a stage: four q of a row i, or four i of a q.  Its values of R: every eighth rank of a q, or
    // a rank of several q.  Pointers are walked from stage to stage.
    const uint32_t li = kQMajor ? (tid & 15u) * 4 : (lane >> 2) + 8 * (warp >> 1), lq = kQMajor ? tid >> 4 : ((lane & 3u) + 4 * (warp & 1u)) * 4;
    const uint64_t I = job.I, Q = job.Q;
    const bool r_j_major = job.r_j_major, l_vec = job.l_vec;
    const TL *lp = static_cast<const TL *>(job.l) + (kQMajor ? (q0 + lq) * I + i0 + li : (i0 + li) * Q + q0 + lq);
    const uint64_t l_next = kQMajor ? 16 * I : 32 * Q, l_step = kQMajor ? kThinQ * I : kThinQ;
    const uint32_t l_have[2] = {(uint32_t)min(i0 + li < I ? I - i0 - li : 0, (uint64_t)4), (uint32_t)(i0 + li + 32 < I)};  // (the second: of rows)
    const uint32_t rj = r_j_major ? tid / kThinQ : tid % kJ, rq = r_j_major ? tid % kThinQ : tid / kJ;
    const uint32_t rj_next = r_j_major ? 256 / kThinQ : 0, rq_next = r_j_major ? 0 : 256 / kJ, ranks = p.rank - j0;
    const TR *rp = static_cast<const TR *>(job.r) + (r_j_major ? (uint64_t)(j0 + rj) * Q + q0 + rq : (q0 + rq) * p.rank + j0 + rj);
    const uint64_t r_next = r_j_major ? rj_next * Q : (uint64_t)rq_next * p.rank, r_step = r_j_major ? kThinQ : (uint64_t)kThinQ * p.rank;
    ptx::pdl_wait();
    ptx::pdl_launch_dependents();

    float4 vl[2];
    float vr[kEach];
    auto load = [&](uint32_t left) {  // the next stage, of which `left` q are there
        #pragma unroll
        for (uint32_t u = 0; u < 2; ++u) {
            const uint32_t n = kQMajor ? (lq + 16 * u < left ? l_have[0] : 0u) : (l_have[u] && lq < left) ? left - lq : 0u;
            vl[u] = load_four(lp + u * l_next, l_vec, n);
        }
        #pragma unroll
        for (uint32_t n = 0; n < kEach; ++n)
            vr[n] = rj + n * rj_next < ranks && rq + n * rq_next < left ? to_f32<TR>(rp[n * r_next]) : 0.0f;
        lp += l_step;
        rp += r_step;
    };
    auto store = [&](float *ls, float *rs) {
        #pragma unroll
        for (uint32_t u = 0; u < 2; ++u) {
            if (kQMajor) {
                *reinterpret_cast<float4 *>(ls + (lq + 16 * u) * kThinPitch + li) = vl[u];
            } else {
                const float f[4] = {vl[u].x, vl[u].y, vl[u].z, vl[u].w};
                #pragma unroll
                for (uint32_t e = 0; e < 4; ++e) ls[(lq + e) * kThinPitch + li + 32 * u] = f[e];
            }
        }
        #pragma unroll
        for (uint32_t n = 0; n < kEach; ++n) {
            rs[(rq + n * rq_next) * kRs + rj + n * rj_next] = vr[n];
        }
    };
    const uint32_t group = tid / kTile, ti = tid % kTile / (kJ / 4) * 4, tj = tid % (kJ / 4) * 4;
    float acc[4][4] = {}, part[4][4] = {};
    uint32_t turn = 0;
    auto left = [&](uint64_t q) { return (uint32_t)min(q < q1 ? q1 - q : 0, (uint64_t)kThinQ); };
    load(left(q0));
    for (uint64_t q = q0; q < q1; q += kThinQ, ++turn) {
        float *const ls = smem + (turn & 1u) * kThinQ * (kThinPitch + kRs), *const rs = ls + kThinQ * kThinPitch;
        store(ls, rs);
        __syncthreads();  // (the place's values of two stages before have been used: their barrier was the last one)
        if (q + kThinQ < q1) load(left(q + kThinQ));
        #pragma unroll
        for (uint32_t n = 0; n < kOwn; ++n) {
            const uint32_t k = group * kOwn + n;
            const float4 a = *reinterpret_cast<const float4 *>(ls + k * kThinPitch + ti), b = *reinterpret_cast<const float4 *>(rs + k * kRs + tj);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
            #pragma unroll
            for (int i = 0; i < 4; ++i)
                #pragma unroll
                for (int j = 0; j < 4; ++j) part[i][j] = fmaf(av[i], bv[j], part[i][j]);
        }
        if (turn % kGroups == kGroups - 1 || q + kThinQ >= q1) {
            #pragma unroll
            for (int i = 0; i < 4; ++i)
                #pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] += part[i][j];
                    part[i][j] = 0.0f;
                }
        }
    }
    // the groups' sums, in order
    __syncthreads();
    #pragma unroll
    for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4 *>(smem + (group * kThinI + ti + i) * kRs + tj) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    if (kGroups > 1) {
        __syncthreads();
        for (uint32_t at = tid; at < kThinI * kJ; at += 256) {
            float v = 0.0f;
            #pragma unroll
            for (uint32_t g = 0; g < kGroups; ++g) v += smem[(g * kThinI + at / kJ) * kRs + at % kJ];
            s_sum[at / kJ * kRs + at % kJ] = v;
        }
    }
    cluster.sync();
    // the CTAs' sums, each CTA a share of the tile's i: j fastest for [I][rank], i for [rank][I]
    const uint32_t per = kThinI / cn;
    for (uint32_t at = tid; at < per * kJ; at += 256) {
        const uint32_t i = rank_in * per + (job.out_j_major ? at % per : at / kJ), j = job.out_j_major ? at / per : at % kJ;
        if (i0 + i >= job.I || j0 + j >= p.rank) continue;
        float v = 0.0f;
        #pragma unroll 4
        for (uint32_t c = 0; c < cn; ++c) v += cluster.map_shared_rank(s_sum, c)[i * kRs + j];
        static_cast<TO *>(job.out)[job.out_j_major ? (j0 + j) * job.I + i0 + i : (i0 + i) * p.rank + j0 + j] = from_f32<TO>(__fmul_rn(v, job.f));
    }
    cluster.sync();  // the sums have been read, before a CTA leaves
}

// y[m][n] = (sum_j T[m][j] * B(j, n)) * scale; one thread per (m, n), n fastest.
template <class T>
__global__ void __launch_bounds__(256)
lora_tb_kernel(const float *__restrict__ t, const T *__restrict__ b, T *__restrict__ y, uint64_t rows,
               uint64_t d_out, uint64_t ldy, uint32_t rank, float scale, int32_t layout) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * d_out) return;
    const uint64_t m = i / d_out, n = i % d_out;
    float acc = 0.0f;
    for (uint32_t j = 0; j < rank; ++j) acc = fmaf(t[m * rank + j], b_at<T>(b, layout, j, n, d_out, rank), acc);
    y[m * ldy + n] = from_f32<T>(__fmul_rn(acc, scale));
}

// out(k, n) = [W(k, n) +] (sum_j A(k, j) * B(j, n)) * scale, stored in the weight's own orientation
// (flat index = k * d_out + n for IN_OUT, n * d_in + k for OUT_IN); one thread per element.
template <class T, bool MERGE>
__global__ void __launch_bounds__(256)
lora_delta_kernel(const T *__restrict__ a, const T *__restrict__ b, const uint8_t *__restrict__ packed,
                  const float *__restrict__ absmax, const uint8_t *__restrict__ scale_codes,
                  const float *__restrict__ scale_of_scales, float *__restrict__ out, uint64_t d_in,
                  uint64_t d_out, uint32_t rank, float scale, int32_t layout) {
    const uint64_t flat = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (flat >= d_in * d_out) return;
    const uint64_t k = layout == NF4_LAYOUT_OUT_IN ? flat % d_in : flat / d_out;
    const uint64_t n = layout == NF4_LAYOUT_OUT_IN ? flat / d_in : flat % d_out;
    float acc = 0.0f;
    for (uint32_t j = 0; j < rank; ++j)
        acc = fmaf(a_at<T>(a, layout, k, j, d_in, rank), b_at<T>(b, layout, j, n, d_out, rank), acc);
    float v = __fmul_rn(acc, scale);
    if (MERGE) {
        const uint32_t byte = __ldg(packed + (flat >> 1));
        const uint32_t code = (flat & 1u) ? (byte >> 4) : (byte & 15u);
        const uint64_t blk = flat / kBlock;
        const float s = absmax ? __ldg(absmax + blk) : dq_scale(__ldg(scale_codes + blk), __ldg(scale_of_scales));
        v = __fadd_rn(__fmul_rn(__uint_as_float(c_level_bits[code]), s), v);
    }
    out[flat] = v;
}

// y[r][rank * width + c] = gathered[rank][r][c]: the ranks' slabs side by side.  16-byte pieces.
__global__ void __launch_bounds__(256)
place_slabs_kernel(const uint4 *__restrict__ gathered, uint4 *__restrict__ y, uint64_t rows, uint64_t pieces_per_row,
                   uint64_t ldy_pieces, uint32_t world) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t per_rank = rows * pieces_per_row;
    if (i >= per_rank * world) return;
    const uint64_t rk = i / per_rank, rem = i % per_rank, r = rem / pieces_per_row, c = rem % pieces_per_row;
    y[r * ldy_pieces + rk * pieces_per_row + c] = gathered[i];
}

// A rank's columns of its own output, pushed into the same columns of every other rank's output
// over NVLink: 16-byte pieces, plain loads from this GPU's memory and plain stores to the peers'
// (mapped into this process by the host).  A persistent grid walks the pieces; when a CTA is done
// it counts itself out on `done`, and the last one makes the launch's stores visible system-wide
// and, if asked, adds one to every rank's arrival counter (this rank's own included).
struct PushParams {
    const uint4 *src;        // this rank's output at its first column
    uint4 *dest[8];          // the ranks' outputs at the same column (own entry unused)
    uint32_t *arrive[8];
    uint32_t *done;          // a word of scratch, zero at first use, left zero
    uint64_t rows, pieces_per_row, ld_pieces;
    uint32_t world, rank, signal;
};

__global__ void __launch_bounds__(256) push_columns_kernel(const PushParams p) {
    const uint64_t total = p.rows * p.pieces_per_row;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t r = i / p.pieces_per_row, c = i - r * p.pieces_per_row;
        const uint64_t at = r * p.ld_pieces + c;
        const uint4 v = __ldcg(p.src + at);
        for (uint32_t d = 0; d < p.world; ++d)
            if (d != p.rank) p.dest[d][at] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(p.done, 1u) == gridDim.x - 1) {
            *p.done = 0;
            if (p.signal) {
                __threadfence_system();
                for (uint32_t d = 0; d < p.world; ++d) atomicAdd_system(p.arrive[d], 1u);
            }
        }
    }
}

// One or two products of the same kind in one launch.
template <class TL, class TR, class TO, bool kQMajor>
int32_t launch_thin(ThinParams p, uint32_t jobs, cudaStream_t s) {
    auto kernel = p.rank <= 16 ? thin_product_kernel<TL, TR, TO, kQMajor, 16>
                  : p.rank <= 32 ? thin_product_kernel<TL, TR, TO, kQMajor, 32> : thin_product_kernel<TL, TR, TO, kQMajor, 64>;
    const uint32_t kj = p.rank <= 16 ? 16 : p.rank <= 32 ? 32 : 64, chunks = (p.rank + kj - 1) / kj;
    uint64_t tiles = 0, longest = 0;
    for (uint32_t i = 0; i < jobs; ++i) {
        ThinJob &job = p.job[i];
        job.tiles = (job.I + kThinI - 1) / kThinI;
        job.l_vec = (kQMajor ? job.I : job.Q) % 4 == 0 && reinterpret_cast<uintptr_t>(job.l) % (4 * sizeof(TL)) == 0;
        tiles += job.tiles;
        longest = longest > job.Q ? longest : job.Q;
    }
    ClusterRoom room;
    NF4_TRY(cluster_room(reinterpret_cast<const void *>(kernel), 256, 0, &room));
    const uint32_t cn = cluster_ctas(tiles * chunks, longest, 2 * kThinQ, room);
    for (uint32_t i = 0; i < jobs; ++i) p.job[i].share = ((p.job[i].Q + cn - 1) / cn + kThinQ - 1) / kThinQ * kThinQ;
    if (tiles * cn >= (1ull << 31) || chunks >= 65536) return fail(NF4_ERR_UNSUPPORTED, "adapter product: too large");
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(tiles * cn), chunks);
    cfg.blockDim = dim3(256);
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cn;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    count_launch();
    return check_cuda(cudaLaunchKernelEx(&cfg, kernel, p), "thin_product_kernel launch");
}
// T = X F with the factor F(k, j) in either orientation
template <class T>
ThinJob xa_job(const T *x, const T *f, float *t, uint64_t rows, uint64_t d_in, int32_t layout) {
    ThinJob job{};
    job.l = x;
    job.r = f;
    job.out = t;
    job.I = rows;
    job.Q = d_in;
    job.f = 1.0f;
    job.r_j_major = layout == NF4_LAYOUT_OUT_IN;
    return job;
}

template <class T>
int32_t forward_t(const void *x, uint64_t rows, uint64_t d_in, uint64_t d_out, const void *a, const void *b,
                  uint32_t rank, float scale, int32_t layout, void *y, uint64_t ldy, float *t, cudaStream_t s) {
    ThinParams p{};
    p.rank = rank;
    p.job[0] = xa_job<T>(static_cast<const T *>(x), static_cast<const T *>(a), t, rows, d_in, layout);
    NF4_TRY((launch_thin<T, T, float, false>(p, 1, s)));
    lora_tb_kernel<T><<<(unsigned)((rows * d_out + 255) / 256), 256, 0, s>>>(
        t, static_cast<const T *>(b), static_cast<T *>(y), rows, d_out, ldy, rank, scale, layout);
    count_launch();
    return check_cuda(cudaGetLastError(), "lora forward launch");
}

template <class T>
int32_t grads_t(const void *x, const void *gy, const void *a, const void *b, uint64_t rows, uint64_t d_in,
                uint64_t d_out, uint32_t rank, float scale, int32_t layout, void *ga, void *gb, float *t,
                float *u, cudaStream_t s) {
    const T *xx = static_cast<const T *>(x), *gg = static_cast<const T *>(gy);
    // T = x A (as in the forward) and U = grad_y B^T (B read as an "A" of the other orientation)
    const int32_t other = layout == NF4_LAYOUT_OUT_IN ? NF4_LAYOUT_IN_OUT : NF4_LAYOUT_OUT_IN;
    ThinParams p{};
    p.rank = rank;
    p.job[0] = xa_job<T>(xx, static_cast<const T *>(a), t, rows, d_in, layout);
    p.job[1] = xa_job<T>(gg, static_cast<const T *>(b), u, rows, d_out, other);
    NF4_TRY((launch_thin<T, T, float, false>(p, 2, s)));
    // grad_A(k, j) = s sum_m x[m][k] U[m][j];  grad_B(j, n) = s sum_m T[m][j] grad_y[m][n]
    auto job = [&](const T *X, const float *R, void *out, uint64_t P, bool p_major) {
        ThinJob g{};
        g.l = X;
        g.r = R;
        g.out = out;
        g.I = P;
        g.Q = rows;
        g.f = scale;
        g.out_j_major = !p_major;
        return g;
    };
    p.job[0] = job(xx, u, ga, d_in, layout == NF4_LAYOUT_IN_OUT);
    p.job[1] = job(gg, t, gb, d_out, layout == NF4_LAYOUT_OUT_IN);
    return launch_thin<T, float, T, true>(p, 2, s);
}

// ---- NCCL, looked up at run time: the library is not linked against it, so that hosts
// without NCCL can load everything else ----
typedef int (*AllGatherFn)(const void *, void *, size_t, int, void *, cudaStream_t);
typedef const char *(*ErrStrFn)(int);

AllGatherFn nccl_all_gather(ErrStrFn *err) {
    static AllGatherFn fn = nullptr;
    static ErrStrFn efn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *sym = dlsym(RTLD_DEFAULT, "ncclAllGather");  // already loaded by the host (torch, a Rust binding)
        void *esym = dlsym(RTLD_DEFAULT, "ncclGetErrorString");
        if (!sym) {
            void *h = dlopen("libnccl.so.2", RTLD_NOW | RTLD_GLOBAL);
            if (h) {
                sym = dlsym(h, "ncclAllGather");
                esym = dlsym(h, "ncclGetErrorString");
            }
        }
        fn = reinterpret_cast<AllGatherFn>(sym);
        efn = reinterpret_cast<ErrStrFn>(esym);
    });
    *err = efn;
    return fn;
}

}  // namespace

uint64_t lora_workspace_bytes(uint64_t rows, uint32_t rank) { return (rows * rank * 4 + 255) / 256 * 256; }

int32_t lora_forward(const void *x, uint64_t rows, uint64_t d_in, uint64_t d_out, const void *a, const void *b,
                     uint32_t rank, float scale, int32_t layout, int32_t io_dtype, void *y, uint64_t ldy,
                     float *t, cudaStream_t s) {
    if (rows * rank >= (1ull << 40) || rows * d_out >= (1ull << 40))
        return fail(NF4_ERR_UNSUPPORTED, "nf4_lora_forward: shape too large");
    return io_dtype == NF4_DTYPE_F32
               ? forward_t<float>(x, rows, d_in, d_out, a, b, rank, scale, layout, y, ldy, t, s)
               : forward_t<__nv_bfloat16>(x, rows, d_in, d_out, a, b, rank, scale, layout, y, ldy, t, s);
}

int32_t lora_delta(const void *a, const void *b, const uint8_t *packed, const float *absmax,
                   const uint8_t *scale_codes, const float *scale_of_scales, uint64_t d_in, uint64_t d_out,
                   uint32_t rank, float scale, int32_t layout, int32_t io_dtype, float *out, cudaStream_t s) {
    const uint64_t n = d_in * d_out;
    if (n >= (1ull << 40)) return fail(NF4_ERR_UNSUPPORTED, "lora delta: shape too large");
    const unsigned grid = (unsigned)((n + 255) / 256);
    const bool merge = packed != nullptr;
    if (io_dtype == NF4_DTYPE_F32) {
        const float *fa = static_cast<const float *>(a), *fb = static_cast<const float *>(b);
        if (merge) lora_delta_kernel<float, true><<<grid, 256, 0, s>>>(fa, fb, packed, absmax, scale_codes, scale_of_scales, out, d_in, d_out, rank, scale, layout);
        else lora_delta_kernel<float, false><<<grid, 256, 0, s>>>(fa, fb, nullptr, nullptr, nullptr, nullptr, out, d_in, d_out, rank, scale, layout);
    } else {
        const __nv_bfloat16 *ha = static_cast<const __nv_bfloat16 *>(a), *hb = static_cast<const __nv_bfloat16 *>(b);
        if (merge) lora_delta_kernel<__nv_bfloat16, true><<<grid, 256, 0, s>>>(ha, hb, packed, absmax, scale_codes, scale_of_scales, out, d_in, d_out, rank, scale, layout);
        else lora_delta_kernel<__nv_bfloat16, false><<<grid, 256, 0, s>>>(ha, hb, nullptr, nullptr, nullptr, nullptr, out, d_in, d_out, rank, scale, layout);
    }
    count_launch();
    return check_cuda(cudaGetLastError(), "lora delta launch");
}

// grad_A and grad_B of y = x W + s (x A) B with W frozen, on CUDA cores; t and u are [rows][rank] f32 scratch
int32_t lora_grads(const void *x, const void *gy, const void *a, const void *b, uint64_t rows, uint64_t d_in,
                   uint64_t d_out, uint32_t rank, float scale, int32_t layout, int32_t io_dtype, void *ga,
                   void *gb, float *t, float *u, cudaStream_t s) {
    if (rows * rank >= (1ull << 40) || (d_in + d_out) * rank >= (1ull << 40))
        return fail(NF4_ERR_UNSUPPORTED, "lora gradients: shape too large");
    return io_dtype == NF4_DTYPE_F32
               ? grads_t<float>(x, gy, a, b, rows, d_in, d_out, rank, scale, layout, ga, gb, t, u, s)
               : grads_t<__nv_bfloat16>(x, gy, a, b, rows, d_in, d_out, rank, scale, layout, ga, gb, t, u, s);
}

// All-gather of the ranks' [rows, width_bytes] slabs into `gathered` ([world][rows][width_bytes]),
// then the slabs side by side into y ([rows][ldy_bytes]).
int32_t gather_slabs(const void *slab, void *gathered, void *y, uint64_t rows, uint64_t width_bytes,
                     uint64_t ldy_bytes, void *comm, int32_t world, cudaStream_t s) {
    if (width_bytes % 16 != 0 || ldy_bytes % 16 != 0 ||
        ((reinterpret_cast<uintptr_t>(gathered) | reinterpret_cast<uintptr_t>(y)) & 15u))
        return fail(NF4_ERR_INVALID_ARG, "sharded forward: slab widths and buffers must be multiples of 16 bytes");
    ErrStrFn estr = nullptr;
    AllGatherFn ag = nccl_all_gather(&estr);
    if (!ag) return fail(NF4_ERR_UNSUPPORTED, "sharded forward: ncclAllGather not found (is NCCL loaded?)");
    const int rc = ag(slab, gathered, (size_t)(rows * width_bytes), /*ncclUint8*/ 1, comm, s);
    if (rc != 0) return fail(NF4_ERR_CUDA, "ncclAllGather failed: %s", estr ? estr(rc) : "unknown NCCL error");
    const uint64_t pieces = rows * (width_bytes / 16) * (uint64_t)world;
    place_slabs_kernel<<<(unsigned)((pieces + 255) / 256), 256, 0, s>>>(
        static_cast<const uint4 *>(gathered), static_cast<uint4 *>(y), rows, width_bytes / 16, ldy_bytes / 16,
        (uint32_t)world);
    count_launch();
    return check_cuda(cudaGetLastError(), "slab placement launch");
}

int32_t push_columns(void *const *y_full, uint32_t *const *arrive, uint32_t world, uint32_t rank, uint64_t rows,
                     uint64_t width_bytes, uint64_t ldy_bytes, bool signal, uint32_t *done, cudaStream_t s) {
    if (world == 0 || world > 8 || rank >= world) return fail(NF4_ERR_INVALID_ARG, "push_columns: world 1 ... 8, rank inside it");
    if (width_bytes == 0 || width_bytes % 16 != 0 || ldy_bytes % 16 != 0 || ldy_bytes < width_bytes * world)
        return fail(NF4_ERR_INVALID_ARG, "push_columns: the shard's width and the output's pitch must be multiples of 16 bytes");
    if (!done) return fail(NF4_ERR_INVALID_ARG, "push_columns: needs a word of scratch");
    PushParams p{};
    for (uint32_t d = 0; d < world; ++d) {
        if (!y_full[d] || (signal && !arrive[d]))
            return fail(NF4_ERR_INVALID_ARG, "push_columns: null output or counter of rank %u", d);
        uint8_t *base = static_cast<uint8_t *>(y_full[d]) + (size_t)rank * width_bytes;
        if (reinterpret_cast<uintptr_t>(base) & 15u) return fail(NF4_ERR_INVALID_ARG, "push_columns: outputs must be 16-byte aligned");
        p.dest[d] = reinterpret_cast<uint4 *>(base);
        p.arrive[d] = arrive[d];
    }
    p.src = p.dest[rank];
    p.done = done;
    p.rows = rows;
    p.pieces_per_row = width_bytes / 16;
    p.ld_pieces = ldy_bytes / 16;
    p.world = world;
    p.rank = rank;
    p.signal = signal ? 1u : 0u;
    if (rows == 0) return NF4_OK;
    const uint64_t pieces = rows * p.pieces_per_row;
    uint64_t ctas = (pieces + 255) / 256;
    if (ctas > (uint64_t)kNumSMs * 8) ctas = (uint64_t)kNumSMs * 8;
    push_columns_kernel<<<(unsigned)ctas, 256, 0, s>>>(p);
    count_launch();
    return check_cuda(cudaGetLastError(), "push_columns_kernel launch");
}

}  // namespace nf4
