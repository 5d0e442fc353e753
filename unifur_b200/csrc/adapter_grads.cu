// The adapter's gradients for bf16 tensors on the tensor cores:
//   grad_A(k, j) = s sum_m x[m][k] U[m][j],   grad_B(j, n) = s sum_m T[m][j] grad_y[m][n],
// T = x A, U = grad_y B^T from the pre-pass kernel as bf16 high and low halves (their f32 values survive:
// two MMAs per tile).
//
// gradient_kernel: out(p, j) = s sum_m X[m][p] R[m][j] as D[p][j] += X^T R (tcgen05, both operands MN-major as they lie).  A
// CTA takes 128 columns p, 64 ranks and a share of the rows; stages of 64 rows of X and of both halves of R (32 KB) come
// by TMA, six in flight where an SM has one CTA, three where there are more CTAs than SMs and it holds two; one thread asks
// for them and one issues their MMAs.  The CTAs that share a
// tile's rows form a cluster: their sums meet through distributed shared memory, each adds (in rank order) and writes its
// part of the columns.  Both gradients are one launch: the tiles of x with U, then those of grad_y with T.  Bound by reading X
// once and R from the L2 for every 128 columns and, at few columns, by the chain of a load, its stages and that exchange.
// Warp MMAs behind transposing loads, whose pipe was half busy, took 40 us for [2048, 14336] and 17 for [2048, 4096] at
// rank 64; in a launch each these tiles took 21 and 12 us, together 22, and 19.7 with six stages in flight.  (Tiles of 256
// columns and half of the rows, which read R half as often, 22.)
#include <cooperative_groups.h>
#include <cuda_bf16.h>

#include "kernels.cuh"
#include "ptx.cuh"
#include "tmap.cuh"

namespace nf4 {
namespace {

constexpr uint32_t kThreads = 192, kCols = 128, kRowsStage = 64;
constexpr uint32_t kBox = kRowsStage * 128, kStage = 4 * kBox;  // X: two boxes of 64 columns; R: high and low halves
constexpr uint32_t smem_of(uint32_t stages) { return stages * kStage + 1024; }
constexpr uint32_t kSumPitch = 68;                              // floats
static_assert(kCols * kSumPitch * 4 <= 3 * kStage, "the sums reuse the stages");

struct Params {
    __nv_bfloat16 *out[2];        // of x (times U), of grad_y (times T)
    uint32_t P[2], p_major[2];
    uint32_t tiles0;              // tiles of the first
    uint32_t rows, rank, chunks, stages_per_share;
    float scale;
};

template <uint32_t kStages>
__global__ void __launch_bounds__(kThreads, 2)  // (registers for two)
gradient_kernel(const __grid_constant__ CUtensorMap tmap_x0, const __grid_constant__ CUtensorMap tmap_r0, const __grid_constant__ CUtensorMap tmap_x1,
                const __grid_constant__ CUtensorMap tmap_r1, const Params p, const FailureRef failure) {
    namespace cg = cooperative_groups;
    cg::cluster_group cluster = cg::this_cluster();
    extern __shared__ uint8_t smem_any[];
    __shared__ __align__(8) uint64_t s_bars[2 * kStages + 1];
    __shared__ uint32_t s_tmem;
    uint8_t *const smem = smem_any + (1024u - (ptx::smem_addr(smem_any) & 1023u)) % 1024u;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t shares = cluster.num_blocks(), share = cluster.block_rank(), tile = blockIdx.x / shares, chunk = blockIdx.y;
    const uint32_t job = tile < p.tiles0 ? 0u : 1u, p0 = (tile - (job ? p.tiles0 : 0u)) * kCols;
    const uint32_t P = job ? p.P[1] : p.P[0], p_major = job ? p.p_major[1] : p.p_major[0];
    const CUtensorMap *const tmap_x = job ? &tmap_x1 : &tmap_x0, *const tmap_r = job ? &tmap_r1 : &tmap_r0;
    __nv_bfloat16 *const out = job ? p.out[1] : p.out[0];
    const uint32_t st0 = share * p.stages_per_share;
    const uint32_t all = (p.rows + kRowsStage - 1) / kRowsStage;
    const uint32_t nst = st0 < all ? min(p.stages_per_share, all - st0) : 0u;
    const uint32_t base = ptx::smem_addr(smem), full0 = ptx::smem_addr(s_bars), empty0 = full0 + 8 * kStages, acc_bar = empty0 + 8 * kStages;
    const uint32_t ranks = min(64u, p.rank - chunk * 64), n16 = (ranks + 15) / 16 * 16;
    float *sum = reinterpret_cast<float *>(smem);
    if (tid == 0) {
        for (uint32_t s = 0; s < kStages; ++s) {
            ptx::mbar_init(full0 + 8 * s, 1);
            ptx::mbar_init(empty0 + 8 * s, 1);
        }
        ptx::mbar_init(acc_bar, 1);
        ptx::fence_mbar_init();
        ptx::fence_proxy_async();
        ptx::prefetch_tmap(tmap_x);
        ptx::prefetch_tmap(tmap_r);
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_addr(&s_tmem), 64);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before();
    __syncthreads();
    ptx::tc_fence_after();
    const uint32_t acc = s_tmem;
    ptx::pdl_launch_dependents();
    ptx::pdl_wait();
    bool ok = true;
    if (warp == 0) {
        for (uint32_t st = 0; lane == 0 && st < nst; ++st) {
            const uint32_t s = st % kStages, full = full0 + 8 * s, dst = base + s * kStage;
            const int32_t m = (int32_t)((st0 + st) * kRowsStage);
            if (st >= kStages && !ptx::mbar_wait_suspended(empty0 + 8 * s, (st / kStages + 1) & 1u)) {
                ok = false;
                NF4_REPORT_FAILURE(*failure.flag, *failure.host, 12);
                break;
            }
            ptx::mbar_arrive_expect_tx(full, kStage);
            ptx::tma_load_2d(dst, tmap_x, (int32_t)p0, m, full);
            ptx::tma_load_2d(dst + kBox, tmap_x, (int32_t)p0 + 64, m, full);
            ptx::tma_load_2d(dst + 2 * kBox, tmap_r, (int32_t)(chunk * 64), m, full);
            ptx::tma_load_2d(dst + 3 * kBox, tmap_r, (int32_t)((p.chunks + chunk) * 64), m, full);
        }
    } else if (warp == 1) {
        const uint32_t idesc = ptx::f16_idesc(1, 128, n16, true, true);
        for (uint32_t st = 0; st < nst; ++st) {
            const uint32_t s = st % kStages;
            ok = ptx::mbar_wait_suspended(full0 + 8 * s, (st / kStages) & 1u);
            if (!ok) {
                if (lane == 0) NF4_REPORT_FAILURE(*failure.flag, *failure.host, 13);
                break;
            }
            ptx::tc_fence_after();
            if (ptx::elect_one()) {
                const uint64_t a = ptx::sw128_desc(base + s * kStage, kBox), hi = ptx::sw128_desc(base + s * kStage + 2 * kBox),
                               lo = ptx::sw128_desc(base + s * kStage + 3 * kBox);
                #pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {  // sixteen rows: 2 KB
                    ptx::mma_ss_f16(acc, a + 128 * i, hi + 128 * i, idesc, (st | i) != 0);
                    ptx::mma_ss_f16(acc, a + 128 * i, lo + 128 * i, idesc, 1);
                }
                ptx::tc_commit(empty0 + 8 * s);
                if (st + 1 == nst) ptx::tc_commit(acc_bar);
            }
            __syncwarp();
        }
    }
    if (!ok) ptx::let_flights_land();
    __syncwarp();
    __syncthreads();
    if (warp >= 2) {  // a lane a column p; ranks that there are not are zeros
        if (nst && !ptx::mbar_wait_suspended(acc_bar, 0)) {
            if (lane == 0) NF4_REPORT_FAILURE(*failure.flag, *failure.host, 14);
        }
        ptx::tc_fence_after();
        const uint32_t q = warp & 3u;
        #pragma unroll
        for (uint32_t c = 0; c < 64; c += 16) {
            uint32_t v[16];
            ptx::tmem_ld16(acc + ((q * 32) << 16) + c, v);
            ptx::tmem_wait_ld();
            const bool real = c < n16 && nst;
            float4 *dst = reinterpret_cast<float4 *>(sum + (q * 32 + lane) * kSumPitch + c);
            #pragma unroll
            for (int i = 0; i < 4; ++i)
                dst[i] = real ? make_float4(__uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]), __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]))
                              : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
        ptx::tc_fence_before();
    }
    if (shares > 1) cluster.sync();
    else __syncthreads();
    const uint32_t per = kCols / shares, per_log = __ffs(per) - 1, q0 = share * per;  // columns of this CTA's part
    if (shares > 1) {  // (the others read their own parts of this CTA's sums: this one may be overwritten)
        #pragma unroll 2
        for (uint32_t i = tid; i < per * 16; i += kThreads) {
            if ((i & 15u) * 4 >= n16) continue;
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
        const uint32_t q = q0 + (p_major ? i >> 6 : i & (per - 1)), j = p_major ? i & 63u : i >> per_log;
        const uint32_t pp = p0 + q, jj = chunk * 64 + j;
        if (pp < P && j < ranks)
            out[p_major ? (size_t)pp * p.rank + jj : (size_t)jj * P + pp] = __float2bfloat16_rn(__fmul_rn(sum[q * kSumPitch + j], p.scale));
    }
    if (shares > 1) cluster.sync();  // the sums have been read, before a CTA leaves
    else __syncthreads();
    if (warp == 1) {
        ptx::tc_fence_after();
        ptx::tmem_dealloc(acc, 64);
    }
}

uint32_t chunks_of(uint32_t rank) { return (rank + 63) / 64; }
uint64_t up256(uint64_t v) { return (v + 255) / 256 * 256; }
uint64_t intermediate_bytes(uint64_t rows, uint32_t rank) { return up256(rows * 2 * 64 * chunks_of(rank) * 2); }
uint64_t tiles_of(uint64_t P) { return (P + kCols - 1) / kCols; }
// ga (p-major as `ga_p_major`) of x [rows][d_in] and u, gb of gy [rows][d_out] and t
int32_t gradients(const void *x, const void *u, void *ga, bool ga_p_major, uint64_t d_in, const void *gy, const void *t, void *gb, bool gb_p_major,
                  uint64_t d_out, uint64_t rows, uint32_t rank, float scale, cudaStream_t s) {
    Params p{};
    p.out[0] = static_cast<__nv_bfloat16 *>(ga);
    p.out[1] = static_cast<__nv_bfloat16 *>(gb);
    p.P[0] = (uint32_t)d_in;
    p.P[1] = (uint32_t)d_out;
    p.p_major[0] = ga_p_major;
    p.p_major[1] = gb_p_major;
    p.rows = (uint32_t)rows;
    p.rank = rank;
    p.chunks = chunks_of(rank);
    p.scale = scale;
    p.tiles0 = (uint32_t)tiles_of(d_in);
    const uint64_t tiles = tiles_of(d_in) + tiles_of(d_out);
    // Shares of the rows: as many as the chip holds clusters for at once, where a share keeps four stages (256 rows)
    ClusterRoom room;
    NF4_TRY(cluster_room(reinterpret_cast<const void *>(gradient_kernel<6>), kThreads, smem_of(6), &room));
    const uint32_t shares = cluster_ctas(tiles, rows, 4 * kRowsStage, room);
    // Three stages in flight leave room for a second CTA on an SM, six ask for what one SM's port brings: columns of 128 in all,
    // 144 tiles of 2048 rows 22.0 and 19.5 us, 64 of 4096 14.0 and 12.8, but 251 tiles of 1100 rows 18.9 and 26.3.
    const bool deep = tiles * shares * p.chunks <= kNumSMs;
    const uint32_t all = (uint32_t)((rows + kRowsStage - 1) / kRowsStage);
    p.stages_per_share = (all + shares - 1) / shares;
    if (tiles * shares >= (1ull << 31)) return fail(NF4_ERR_UNSUPPORTED, "gradients: too many columns");
    CUtensorMap map_x0, map_r0, map_x1, map_r1;
    const uint64_t ld_r = 2 * 64 * (uint64_t)p.chunks;
    auto of = [&](CUtensorMap *map, const void *v, uint64_t cols) {
        return make_map(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, v, rows, cols, cols * 2, kRowsStage, 64, CU_TENSOR_MAP_SWIZZLE_128B);
    };
    NF4_TRY(of(&map_x0, x, d_in));
    NF4_TRY(of(&map_r0, u, ld_r));
    NF4_TRY(of(&map_x1, gy, d_out));
    NF4_TRY(of(&map_r1, t, ld_r));
    FailureRef failure;
    NF4_TRY(prefill_failure_ref(&failure));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(tiles * shares), p.chunks);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem_of(deep ? 6 : 3);
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
    auto kernel = deep ? gradient_kernel<6> : gradient_kernel<3>;
    if (!deep) NF4_TRY(cluster_room(reinterpret_cast<const void *>(kernel), kThreads, smem_of(3), &room));
    return check_cuda(cudaLaunchKernelEx(&cfg, kernel, map_x0, map_r0, map_x1, map_r1, p, failure), "gradient_kernel launch");
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
    return gradients(x, u, ga, in_out, d_in, gy, t, gb, !in_out, d_out, rows, rank, scale, s);
}

}  // namespace nf4
