// The adapter's gradients for bf16 tensors on warp MMAs:
//   grad_A(k, j) = s sum_m x[m][k] U[m][j],   grad_B(j, n) = s sum_m T[m][j] grad_y[m][n],
// T = x A, U = grad_y B^T from the pre-pass kernel as bf16 high and low halves (their f32 values survive:
// two MMAs per tile).
//
// gradient_kernel: out(p, j) = s sum_m X[m][p] R[m][j] as D[p][j] += A[p][m] B[m][j] (m16n8k16).  A CTA takes
// 128 columns p, 64 ranks and a share of the rows; 64 rows of X and R per stage come by 16-byte
// asynchronous copies, three stages in flight, and both operands are transposing matrix loads of what lies
// there.  Eight warps: four pieces of 32 columns, two halves of a stage's rows.  The CTAs that share a tile's
// rows form a cluster: their sums meet through distributed shared memory, each adds (in rank order) and writes its part
// of the columns.  Bound by reading X once and, at few columns, by the chain of a load, its stages and that
// exchange; sums through the workspace, added by the CTA that arrived last, took 25 us for [2048, 4096] (now
// 17) and 45 for [2048, 14336] (now 40) at rank 64.
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "kernels.cuh"
#include "ptx.cuh"

namespace nf4 {
namespace {

constexpr uint32_t kThreads = 256, kCols = 128, kRowsStage = 64, kStages = 3;
constexpr uint32_t kPitch = 272;                           // 256 bytes of a row and 16 of padding
constexpr uint32_t kXStage = kRowsStage * kPitch, kStage = 2 * kXStage;
constexpr uint32_t kSumPitch = 68;                         // floats
static_assert(kCols * kSumPitch * 4 <= kStages * kStage, "the sums reuse the stages");

struct Params {
    const __nv_bfloat16 *x, *r;   // [rows][P]; [rows][2 * 64 * chunks]: hi halves, then lo
    __nv_bfloat16 *out;
    uint32_t rows, P, rank, chunks, stages_per_share, p_major;
    float scale;
};

__global__ void __launch_bounds__(kThreads, 2) gradient_kernel(const Params p) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ __align__(16) uint8_t smem[];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t g = lane >> 2, t = lane & 3u, li = lane >> 3, lr = lane & 7u;
    const uint32_t pw = warp & 3u, h = warp >> 2;
    const uint32_t shares = cluster.num_blocks(), share = cluster.block_rank(), p0 = blockIdx.x / shares * kCols;
    const uint32_t st0 = share * p.stages_per_share;
    const uint32_t all = (p.rows + kRowsStage - 1) / kRowsStage;
    const uint32_t nst = st0 < all ? min(p.stages_per_share, all - st0) : 0u;
    const uint32_t base = ptx::smem_addr(smem), ld_r = 128 * p.chunks;
    float *sum = reinterpret_cast<float *>(smem);
    ptx::pdl_launch_dependents();
    ptx::pdl_wait();
    for (uint32_t chunk = 0; chunk < p.chunks; ++chunk) {
        const uint32_t ranks = min(64u, p.rank - chunk * 64), tiles16 = (ranks + 15) / 16;
        auto load = [&](uint32_t st) {
            if (st < nst) {
                const uint32_t m0 = (st0 + st) * kRowsStage, dst = base + (st % kStages) * kStage;
                #pragma unroll
                for (uint32_t q = 0; q < 4; ++q) {  // X: 64 rows x 16 pieces of eight columns
                    const uint32_t i = tid + q * kThreads, r = i >> 4, c = i & 15u;
                    const bool real = m0 + r < p.rows && p0 + c * 8 < p.P;
                    ptx::cp_async_16_or_zero(dst + r * kPitch + c * 16, p.x + (real ? (size_t)(m0 + r) * p.P + p0 + c * 8 : 0), real);
                }
                #pragma unroll
                for (uint32_t q = 0; q < 4; ++q) {  // R: 64 rows x (8 pieces of hi, 8 of lo)
                    const uint32_t i = tid + q * kThreads, r = i >> 4, c = i & 15u;
                    if ((c & 7u) >= 2 * tiles16) continue;
                    const bool real = m0 + r < p.rows;
                    const size_t at = (size_t)(m0 + r) * ld_r + (c >> 3) * 64 * p.chunks + chunk * 64 + (c & 7u) * 8;
                    ptx::cp_async_16_or_zero(dst + kXStage + r * kPitch + c * 16, p.r + (real ? at : 0), real);
                }
            }
            ptx::cp_async_commit();
        };
        float acc[2][8][4];
        #pragma unroll
        for (int a = 0; a < 2; ++a)
            #pragma unroll
            for (int u = 0; u < 8; ++u) acc[a][u][0] = acc[a][u][1] = acc[a][u][2] = acc[a][u][3] = 0.0f;
        load(0);
        load(1);
        for (uint32_t st = 0; st < nst; ++st) {
            ptx::cp_async_wait<1>();
            __syncthreads();
            load(st + 2);
            const uint32_t xs = base + (st % kStages) * kStage, rs = xs + kXStage;
            #pragma unroll
            for (uint32_t k2 = 0; k2 < 2; ++k2) {
                const uint32_t m = (2 * h + k2) * 16;
                uint32_t af[2][4];
                #pragma unroll
                for (int a = 0; a < 2; ++a)
                    ptx::ldmatrix_x4_trans(af[a], xs + (m + (li >> 1) * 8 + lr) * kPitch + (pw * 32 + a * 16 + (li & 1u) * 8) * 2);
                const uint32_t b_at = rs + (m + (li & 1u) * 8 + lr) * kPitch + (li >> 1) * 16;
                #pragma unroll
                for (uint32_t u = 0; u < 4; ++u) {
                    if (u >= tiles16) break;
                    #pragma unroll
                    for (uint32_t half = 0; half < 2; ++half) {  // hi, then lo
                        uint32_t bf[4];
                        ptx::ldmatrix_x4_trans(bf, b_at + half * 128 + u * 32);
                        #pragma unroll
                        for (int a = 0; a < 2; ++a) {
                            ptx::mma_16816_bf16(acc[a][2 * u], af[a][0], af[a][1], af[a][2], af[a][3], bf[0], bf[1]);
                            ptx::mma_16816_bf16(acc[a][2 * u + 1], af[a][0], af[a][1], af[a][2], af[a][3], bf[2], bf[3]);
                        }
                    }
                }
            }
        }
        ptx::cp_async_wait<0>();
        // the two halves of the rows, in order
        for (uint32_t turn = 0; turn < 2; ++turn) {
            __syncthreads();
            if (h == turn) {
                #pragma unroll
                for (int a = 0; a < 2; ++a)
                    #pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        float2 *lo = reinterpret_cast<float2 *>(sum + (pw * 32 + a * 16 + g) * kSumPitch + u * 8 + 2 * t);
                        float2 *hi = reinterpret_cast<float2 *>(sum + (pw * 32 + a * 16 + g + 8) * kSumPitch + u * 8 + 2 * t);
                        const float2 l = turn ? *lo : make_float2(0.0f, 0.0f), hh = turn ? *hi : make_float2(0.0f, 0.0f);
                        *lo = make_float2(l.x + acc[a][u][0], l.y + acc[a][u][1]);
                        *hi = make_float2(hh.x + acc[a][u][2], hh.y + acc[a][u][3]);
                    }
            }
        }
        if (shares > 1) cluster.sync();
        else __syncthreads();
        const uint32_t per = kCols / shares, per_log = __ffs(per) - 1, q0 = share * per;  // columns of this CTA's part
        if (shares > 1) {  // (the others read their own parts of this CTA's sums: this one may be overwritten)
            #pragma unroll 2
            for (uint32_t i = tid; i < per * 16; i += kThreads) {
                if ((i & 15u) >= 4 * tiles16) continue;
                const uint32_t at = (q0 + (i >> 4)) * kSumPitch + (i & 15u) * 4;
                float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                #pragma unroll 8
                for (uint32_t c = 0; c < shares; ++c) {
                    const float4 o = *reinterpret_cast<const float4 *>(cluster.map_shared_rank(sum, c) + at);
                    v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
                }
                *reinterpret_cast<float4 *>(sum + at) = v;
            }
            __syncthreads();
        }
        for (uint32_t i = tid; i < per * 64; i += kThreads) {
            // p fastest for [rank][P] outputs, j fastest for [P][rank]
            const uint32_t q = q0 + (p.p_major ? i >> 6 : i & (per - 1)), j = p.p_major ? i & 63u : i >> per_log;
            const uint32_t pp = p0 + q, jj = chunk * 64 + j;
            if (pp < p.P && j < ranks)
                p.out[p.p_major ? (size_t)pp * p.rank + jj : (size_t)jj * p.P + pp] = __float2bfloat16_rn(__fmul_rn(sum[q * kSumPitch + j], p.scale));
        }
        if (shares > 1) cluster.sync();
        else __syncthreads();  // the sums have been read (before the next chunk's stages, and before a CTA leaves)
    }
}

uint32_t chunks_of(uint32_t rank) { return (rank + 63) / 64; }
uint64_t up256(uint64_t v) { return (v + 255) / 256 * 256; }
uint64_t intermediate_bytes(uint64_t rows, uint32_t rank) { return up256(rows * 2 * 64 * chunks_of(rank) * 2); }
uint64_t tiles_of(uint64_t P) { return (P + kCols - 1) / kCols; }
int32_t gradient(const void *x, const void *r, void *out, uint64_t rows, uint64_t P, uint32_t rank, float scale, bool p_major,
                 cudaStream_t s) {
    Params p{};
    p.x = static_cast<const __nv_bfloat16 *>(x);
    p.r = static_cast<const __nv_bfloat16 *>(r);
    p.out = static_cast<__nv_bfloat16 *>(out);
    p.rows = (uint32_t)rows;
    p.P = (uint32_t)P;
    p.rank = rank;
    p.chunks = chunks_of(rank);
    // Shares of the rows: as many as the chip holds clusters for at once, where a share keeps four stages (256 rows)
    const void *kernel = reinterpret_cast<const void *>(gradient_kernel);
    ClusterRoom room;
    NF4_TRY(cluster_room(kernel, kThreads, kStages * kStage, &room));
    const uint32_t shares = cluster_ctas(tiles_of(P), rows, 4 * kRowsStage, room);
    const uint32_t all = (uint32_t)((rows + kRowsStage - 1) / kRowsStage);
    p.stages_per_share = (all + shares - 1) / shares;
    p.p_major = p_major;
    p.scale = scale;
    if (tiles_of(P) * shares >= (1ull << 31)) return fail(NF4_ERR_UNSUPPORTED, "gradient: too many columns");
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(tiles_of(P) * shares));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kStages * kStage;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = shares;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = shares > 1 ? 2 : 1;
    count_launch();
    return check_cuda(cudaLaunchKernelEx(&cfg, gradient_kernel, p), "gradient_kernel launch");
}

}  // namespace

bool adapter_grads_supported(const void *x, const void *gy, const void *a, const void *b, uint64_t rows, uint64_t d_in,
                             uint64_t d_out, uint32_t rank) {
    return d_in % 8 == 0 && d_out % 8 == 0 && rows < (1ull << 31) && d_in < (1ull << 31) && d_out < (1ull << 31) && rank <= 4096 &&
           aligned16(x) && aligned16(gy) && (reinterpret_cast<uintptr_t>(a) & 1u) == 0 && (reinterpret_cast<uintptr_t>(b) & 1u) == 0;
}

// T | U
uint64_t adapter_grads_bytes(uint64_t rows, uint64_t, uint64_t, uint32_t rank) {
    return rank ? 2 * intermediate_bytes(rows, rank) : 0;
}

void *adapter_grads_u(void *scratch, uint64_t rows, uint32_t rank) {
    return static_cast<uint8_t *>(scratch) + intermediate_bytes(rows, rank);
}

int32_t adapter_grads(const void *x, const void *gy, const void *a, const void *b, uint64_t rows, uint64_t d_in,
                      uint64_t d_out, uint32_t rank, float scale, int32_t layout, void *ga, void *gb, void *scratch,
                      bool u_ready, cudaStream_t s) {
    const bool in_out = layout == NF4_LAYOUT_IN_OUT;
    void *t = scratch, *u = adapter_grads_u(scratch, rows, rank);
    PrepassArgs q{};
    q.M = (uint32_t)rows;
    q.rank = rank;
    if (!u_ready) {  // U = grad_y B^T, B [d_out][r] or [r][d_out]
        q.x = gy;
        q.K = (uint32_t)d_out;
        q.a = b;
        q.k_major = !in_out;
        q.r_out = u;
        NF4_TRY(activations_prepass(q, s));
    }
    q.x = x;             // T = x A, A [r][d_in] or [d_in][r]
    q.K = (uint32_t)d_in;
    q.a = a;
    q.k_major = in_out;
    q.r_out = t;
    NF4_TRY(activations_prepass(q, s));
    NF4_TRY(gradient(x, u, ga, rows, d_in, rank, scale, in_out, s));
    return gradient(gy, t, gb, rows, d_out, rank, scale, !in_out, s);
}

}  // namespace nf4
