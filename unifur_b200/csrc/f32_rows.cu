// f32 tensors at up to 16 rows with W [d_out, d_in] (the reference's tensor type on the measured
// layout): the decode kernels take bf16 activations, and rounding f32 activations to bf16 would cost
// 1e-3 by itself.  So each row is split into two bf16 rows, x = hi + lo (sixteen bits of mantissa
// between them), the decode kernel multiplies the 2 m rows with f32 outputs, and one more kernel
// adds the two halves, the bias and the adapter term s (x A^T) B^T, which is computed in f32 from
// the f32 factors as the reference does.  At most eight rows per pass (sixteen for the kernel).
// 9 x 9728 x 18240 at rank 32: 160 us with T by CTAs of many columns (38 of it) and a thread per output that walked its row of B
// value by value (29), now 108; 4 x 4096 x 11008 at rank 16 28.7, now 16.7; 16 x 4096 x 4096 at rank 64 54.6, now 34.9.
#include <cuda_bf16.h>

#include "kernels.cuh"
#include "ptx.cuh"

namespace nf4 {
namespace {

__global__ void __launch_bounds__(256)
split_rows_kernel(const float *__restrict__ x, __nv_bfloat16 *__restrict__ xs, uint32_t m, uint64_t K) {
    ptx::pdl_wait();
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (uint64_t)m * K) return;
    const float v = x[i];
    const __nv_bfloat16 hi = __float2bfloat16_rn(v);
    float rest = v - __bfloat162float(hi);
    if (!(fabsf(v) < 3.0e38f)) rest = 0.0f;  // infinities and NaNs travel in the high part alone
    xs[i] = hi;
    xs[(uint64_t)m * K + i] = __float2bfloat16_rn(rest);
}

// y[r][n] = yy[r][n] + yy[m + r][n] (+ bias[n]) (+ scale * sum_j t[r][j] * B[n][j]).  A thread has a column n of two
// rows: its row of B is read four values at a time where they are whole (`wide`), T comes from shared memory.
constexpr uint32_t kCombineThreads = 128, kPassRows = 8, kThreadRows = 2, kCombineCols = kCombineThreads / (kPassRows / kThreadRows), kMaxRankHeld = 256;
__global__ void __launch_bounds__(kCombineThreads)
combine_rows_kernel(const float *__restrict__ yy, const float *__restrict__ bias, const float *__restrict__ t,
                    const float *__restrict__ b, float *__restrict__ y, uint32_t m, uint64_t N, uint64_t ldy,
                    uint32_t rank, float scale, bool wide) {
    __shared__ float s_t[kPassRows * kMaxRankHeld];
    const bool held = rank <= kMaxRankHeld;
    for (uint32_t i = threadIdx.x; held && i < m * rank; i += kCombineThreads) s_t[i] = t[i];
    __syncthreads();
    const float *tt = held ? s_t : t;
    const uint64_t n = (uint64_t)blockIdx.x * kCombineCols + threadIdx.x % kCombineCols;
    const uint32_t r0 = threadIdx.x / kCombineCols * kThreadRows;
    if (n >= N || r0 >= m) return;
    float acc[kThreadRows] = {};
    uint32_t j = 0;
    #pragma unroll 4
    for (; wide && j + 4 <= rank; j += 4) {
        const float4 v = __ldg(reinterpret_cast<const float4 *>(b + n * rank + j));
        #pragma unroll
        for (uint32_t r = 0; r < kThreadRows; ++r) {
            const float *row = tt + min(r0 + r, m - 1) * rank + j;
            acc[r] = fmaf(row[3], v.w, fmaf(row[2], v.z, fmaf(row[1], v.y, fmaf(row[0], v.x, acc[r]))));
        }
    }
    for (; j < rank; ++j) {
        const float v = __ldg(b + n * rank + j);
        #pragma unroll
        for (uint32_t r = 0; r < kThreadRows; ++r) acc[r] = fmaf(tt[min(r0 + r, m - 1) * rank + j], v, acc[r]);
    }
    const float add = bias ? __ldg(bias + n) : 0.0f;
    #pragma unroll
    for (uint32_t i = 0; i < kThreadRows; ++i) {
        const uint32_t r = r0 + i;
        if (r >= m) break;
        float v = yy[r * N + n] + yy[(uint64_t)(m + r) * N + n];
        if (rank) v += __fmul_rn(acc[i], scale);
        y[r * ldy + n] = bias ? v + add : v;
    }
}

inline uint64_t up256(uint64_t v) { return (v + 255) / 256 * 256; }

struct Scratch {
    uint64_t off_xs, off_yy, off_t, bytes;
};
Scratch scratch_layout(uint64_t d_in, uint64_t d_out, uint32_t rank) {
    Scratch s;
    const uint64_t a = decode_workspace_bytes(16, d_in, d_out, 0), b = decode2_workspace_bytes(16, d_in, d_out, 0);
    s.off_xs = up256(a > b ? a : b);
    if (s.off_xs < 256) s.off_xs = 256;
    s.off_yy = s.off_xs + up256(16 * d_in * 2);
    s.off_t = s.off_yy + up256(16 * d_out * 4);
    s.bytes = s.off_t + up256(16ull * rank * 4);
    return s;
}

// the bf16 call one pass makes: 2 m rows, f32 outputs, no bias, no adapter
nf4_linear_args halves_args(const nf4_linear_args &a, uint64_t m, const void *xs, void *yy) {
    nf4_linear_args h = a;
    h.io_dtype = NF4_DTYPE_BF16;
    h.y_f32 = 1;
    h.rows = 2 * m;
    h.x = xs;
    h.y = yy;
    h.ldy = a.d_out;
    h.bias = nullptr;
    h.lora_a = h.lora_b = nullptr;
    h.lora_rank = 0;
    h.lora_scale = 0.0f;
    return h;
}

}  // namespace

uint64_t f32_rows_workspace_bytes(uint64_t rows, uint64_t d_in, uint64_t d_out, uint32_t lora_rank) {
    if (rows == 0 || rows > 16) return 0;
    return scratch_layout(d_in, d_out, lora_rank).bytes;
}

bool f32_rows_supported(const nf4_linear_args &a) {
    if (a.layout != NF4_LAYOUT_OUT_IN || a.io_dtype != NF4_DTYPE_F32 || a.rows == 0 || a.rows > 16) return false;
    if (!a.workspace || (reinterpret_cast<uintptr_t>(a.workspace) & 255u)) return false;
    const Scratch sc = scratch_layout(a.d_in, a.d_out, a.lora_a ? a.lora_rank : 0);
    if (a.workspace_bytes < sc.bytes) return false;
    uint8_t *ws = static_cast<uint8_t *>(a.workspace);
    const nf4_linear_args h = halves_args(a, a.rows < 8 ? a.rows : 8, ws + sc.off_xs, ws + sc.off_yy);
    return decode_supported(h) || decode2_supported(h);
}

int32_t f32_rows_forward(const nf4_linear_args &a, cudaStream_t stream) {
    if (!f32_rows_supported(a)) return fail(NF4_ERR_UNSUPPORTED, "f32_rows_forward: unsupported shape");
    const uint32_t rank = a.lora_a ? a.lora_rank : 0;
    const Scratch sc = scratch_layout(a.d_in, a.d_out, rank);
    uint8_t *ws = static_cast<uint8_t *>(a.workspace);
    __nv_bfloat16 *xs = reinterpret_cast<__nv_bfloat16 *>(ws + sc.off_xs);
    float *yy = reinterpret_cast<float *>(ws + sc.off_yy);
    float *t = reinterpret_cast<float *>(ws + sc.off_t);
    const uint64_t ldy = a.ldy ? a.ldy : a.d_out;
    const float *x = static_cast<const float *>(a.x);
    float *y = static_cast<float *>(a.y);
    if (rank)  // T = x A^T for all the rows, in f32
        NF4_TRY(small_lora_t(a.x, a.lora_a, t, a.rows, a.d_in, rank, true, true, stream));
    for (uint64_t r0 = 0; r0 < a.rows; r0 += kPassRows) {
        const uint32_t m = (uint32_t)(a.rows - r0 < kPassRows ? a.rows - r0 : kPassRows);
        count_launch();
        NF4_TRY(launch_maybe_overlapped(split_rows_kernel, dim3((unsigned)((m * a.d_in + 255) / 256)), dim3(256), 0, stream, true, x + r0 * a.d_in, xs,
                                        m, a.d_in));
        nf4_linear_args h = halves_args(a, m, xs, yy);
        h.workspace_bytes = sc.off_xs;
        if (decode_supported(h)) NF4_TRY(decode_forward(h, stream));
        else NF4_TRY(decode2_forward(h, stream));
        // (an ordinary launch: as the decode kernel's programmatic dependent this one took 16 x 4096 x 4096 from 35 to 70 us)
        const bool wide = rank % 4 == 0 && aligned16(a.lora_b);
        count_launch();
        NF4_TRY(launch_maybe_overlapped(combine_rows_kernel, dim3((unsigned)((a.d_out + kCombineCols - 1) / kCombineCols)), dim3(kCombineThreads), 0,
                                        stream, false, static_cast<const float *>(yy), a.bias, static_cast<const float *>(t + r0 * rank),
                                        static_cast<const float *>(a.lora_b), y + r0 * ldy, m, a.d_out, ldy, rank, a.lora_scale, wide));
    }
    return NF4_OK;
}

}  // namespace nf4
