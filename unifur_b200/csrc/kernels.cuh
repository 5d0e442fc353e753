// Internal kernel-launcher interface between the C ABI (api.cu) and the kernel files.
#pragma once
#include "nf4_common.cuh"

namespace nf4 {

// Launch `kernel` so that it may start while its predecessor in `stream` is still running
// (programmatic dependent launch); the kernel must call ptx::pdl_wait() before it touches
// anything the predecessor writes.  Falls back to an ordinary launch when `overlap` is false.
template <class... KArgs, class... Args>
int32_t launch_maybe_overlapped(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                cudaStream_t stream, bool overlap, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = overlap ? 1 : 0;
    return check_cuda(cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...), "kernel launch");
}
// api.cu: sets cudaFuncAttributeMaxDynamicSharedMemorySize for `kernel` on the current device,
// once per (kernel, device): the attribute belongs to the device a kernel is loaded on.
int32_t ensure_dynamic_smem(const void *kernel, int bytes);

// api.cu: how many clusters of 2^i CTAs (`any`: of i CTAs) of `kernel` the current device holds at once, by the driver's
// count (once per kernel and device; 0: it has no place for one).  Sets the kernel's dynamic shared memory, and allows it clusters
// of sixteen.  (A whole B200, two CTAs of 108 KB on an SM: 148 of two, 71 of four, 33 of eight, 14 of sixteen.)
constexpr uint32_t kClusterSizes = 5;
struct ClusterRoom {
    uint32_t of[kClusterSizes];
    uint32_t any[(1u << (kClusterSizes - 1)) + 1];
};
int32_t cluster_room(const void *kernel, uint32_t threads, uint32_t smem, ClusterRoom *room);
// CTAs to a cluster when each takes a piece of a tile's `length`: as many as leave the tiles' clusters in one wave and
// every CTA a piece of more than half a unit, 1 at least.
uint32_t cluster_ctas(uint64_t tiles, uint64_t length, uint64_t unit, const ClusterRoom &room);

// lora.cu: the adapter alone, its dense update, the merge, and the gather of column slabs
uint64_t lora_workspace_bytes(uint64_t rows, uint32_t rank);
int32_t lora_forward(const void *x, uint64_t rows, uint64_t d_in, uint64_t d_out, const void *a, const void *b,
                     uint32_t rank, float scale, int32_t layout, int32_t io_dtype, void *y, uint64_t ldy,
                     float *t, cudaStream_t s);
int32_t lora_delta(const void *a, const void *b, const uint8_t *packed, const float *absmax,
                   const uint8_t *scale_codes, const float *scale_of_scales, uint64_t d_in, uint64_t d_out,
                   uint32_t rank, float scale, int32_t layout, int32_t io_dtype, float *out, cudaStream_t s);
int32_t lora_grads(const void *x, const void *gy, const void *a, const void *b, uint64_t rows, uint64_t d_in,
                   uint64_t d_out, uint32_t rank, float scale, int32_t layout, int32_t io_dtype, void *ga,
                   void *gb, float *t, float *u, cudaStream_t s);

// adapter_grads.cu: the same for bf16 tensors on tcgen05.  `scratch` (256-byte aligned) holds R = x a and
// grad_y b in the pre-pass's form; u_ready:
// adapter_grads_u(scratch, ...) already holds grad_y b (the pre-pass of grad_x left it there).
bool adapter_grads_supported(const void *x, const void *gy, const void *a, const void *b, uint64_t rows, uint64_t d_in,
                             uint64_t d_out, uint32_t rank);
uint64_t adapter_grads_bytes(uint64_t rows, uint64_t d_in, uint64_t d_out, uint32_t rank);
void *adapter_grads_u(void *scratch, uint64_t rows, uint32_t rank);
int32_t adapter_grads(const void *x, const void *gy, const void *a, const void *b, uint64_t rows, uint64_t d_in,
                      uint64_t d_out, uint32_t rank, float scale, int32_t layout, void *ga, void *gb, void *scratch,
                      bool u_ready, cudaStream_t s);
int32_t push_columns(void *const *y_full, uint32_t *const *arrive, uint32_t world, uint32_t rank, uint64_t rows,
                     uint64_t width_bytes, uint64_t ldy_bytes, bool signal, uint32_t *done, cudaStream_t s);
int32_t gather_slabs(const void *slab, void *gathered, void *y, uint64_t rows, uint64_t width_bytes,
                     uint64_t ldy_bytes, void *comm, int32_t world, cudaStream_t s);

// quantize.cu
int32_t quantize_packed(const float *values, uint64_t len, uint8_t *packed, float *absmax,
                        cudaStream_t stream);
int32_t quantize_unpacked(const float *values, uint64_t len, uint8_t *codes, float *absmax,
                          cudaStream_t stream);
int32_t dequantize_packed(const uint8_t *packed, uint64_t len, const float *absmax,
                          const uint8_t *scale_codes, const float *scale_of_scales, float *out,
                          cudaStream_t stream);
int32_t dequantize_unpacked(const uint8_t *codes, uint64_t len, const float *absmax,
                            const uint8_t *scale_codes, const float *scale_of_scales, float *out,
                            cudaStream_t stream);
// n_maxima: how many of the largest scales of its CTAs (2 * kNumSMs at most) the kernel leaves in `maxima`, which may be none
int32_t quantize_transposed(const void *src, bool src_bf16, uint64_t rows, uint64_t cols,
                            uint8_t *packed, float *absmax, void *workspace, uint64_t workspace_bytes,
                            cudaStream_t stream, float *maxima = nullptr, uint32_t *n_maxima = nullptr);
uint64_t quantize_transposed_double_workspace_bytes(uint64_t rows, uint64_t cols);
int32_t quantize_transposed_double(const void *src, bool src_bf16, uint64_t rows, uint64_t cols, uint8_t *packed, float *absmax, uint8_t *scale_codes,
                                   float *scale_of_scales, void *workspace, uint64_t workspace_bytes, cudaStream_t stream);
int32_t embedding_gather(const uint8_t *packed, const float *absmax, const uint8_t *scale_codes,
                         const float *scale_of_scales, uint64_t n_embedding, uint64_t d_model,
                         const int64_t *ids, uint64_t n_ids, void *out, bool out_bf16,
                         cudaStream_t stream);
int32_t double_quantize(const float *absmax, uint64_t nblocks, uint8_t *scale_codes,
                        float *scale_of_scales, cudaStream_t stream);
int32_t selfcheck_fast(uint64_t first_bits, uint64_t count, float absmax,
                       unsigned long long *mismatches_dev, cudaStream_t stream);
int32_t selfcheck_codes(uint64_t first_bits, uint64_t count, unsigned long long *mismatches_dev,
                        cudaStream_t stream);

// decode_gemv.cu: rows <= 16, NF4_LAYOUT_OUT_IN, bf16 activations.
bool decode_supported(const nf4_linear_args &a);
uint64_t decode_workspace_bytes(uint64_t rows, uint64_t d_in, uint64_t d_out, uint32_t lora_rank);
// A kernel's failure code goes to its device flag and, where the host has given the kernel's file
// a word of mapped host memory (the host-pointer entry points do, so that they need no copy to
// look at it), to that word as well.
#define NF4_REPORT_FAILURE(flag, host_word, code)                          \
    do {                                                                   \
        atomicExch(&(flag), (code));                                       \
        if (host_word) *reinterpret_cast<volatile int *>(host_word) = (code); \
    } while (0)
int32_t decode_set_host_flag(int *mapped);
int32_t decode2_set_host_flag(int *mapped);
int32_t prefill_set_host_flag(int *mapped);

// api.cu: CTAs a kernel that puts one CTA on every SM may use (the SM count less nf4_reserve_sms)
uint32_t persistent_ctas();
int32_t decode_forward(const nf4_linear_args &a, cudaStream_t stream);
int32_t decode_forward_scatter(const nf4_linear_args &a, void *const *dest, uint32_t *const *arrive, uint32_t world,
                               uint32_t rank, uint64_t ldy, bool signal, uint32_t *wait_on, uint32_t wait_expected,
                               cudaStream_t stream);
int32_t decode_forward_host(const nf4_linear_args &a, const void *x_host, uint32_t *host_done, uint32_t value, cudaStream_t stream, bool *taken);
int32_t decode_peer_wait(uint32_t *counter, uint32_t expected, uint32_t limit_ns, cudaStream_t stream);
int32_t decode_share_plan(uint32_t rows, uint32_t d_in, uint32_t d_out, uint32_t rank, uint32_t cta, uint32_t *out4);
int32_t decode_forward_grouped(const nf4_linear_args *a, uint32_t count, cudaStream_t stream, bool *taken);

int32_t decode_selftest_wait(uint32_t limit_ns, unsigned long long *waited_ns_dev, cudaStream_t stream);
// device addresses (current device) of the kernels' failure flags
int32_t decode_error_flag_ptr(int **dev_ptr);
int32_t decode2_error_flag_ptr(int **dev_ptr);
int32_t prefill_error_flag_ptr(int **dev_ptr);
// where the kernels around the tensor-core GEMM report a failure: its flag and the place of its host word (current device)
struct FailureRef {
    int *flag;
    int **host;
};
int32_t prefill_failure_ref(FailureRef *ref);
uint64_t decode_static_scratch_bytes();
int32_t decode_forward_static_scratch(const nf4_linear_args &a, cudaStream_t stream);

// decode_umma.cu: rows <= 16 through tcgen05 (the fast decode path when its shape rules hold).
bool decode2_supported(const nf4_linear_args &a);
uint64_t decode2_workspace_bytes(uint64_t rows, uint64_t d_in, uint64_t d_out, uint32_t lora_rank);
int32_t decode2_forward(const nf4_linear_args &a, cudaStream_t stream);

// generic_linear.cu: any layout / dtype / shape on CUDA cores (exact f32 weights).
uint64_t generic_workspace_bytes(uint64_t rows, uint64_t d_in, uint64_t d_out, uint32_t lora_rank);
bool generic_reads_flags(const nf4_linear_args &a);
int32_t generic_forward(const nf4_linear_args &a, cudaStream_t stream);

// in_out_strips.cu: NF4_LAYOUT_IN_OUT at few rows (sixteen per launch), d_out a multiple of 64, f32 arithmetic
bool strips_supported(const nf4_linear_args &a);
uint64_t strips_workspace_bytes(uint64_t rows, uint64_t d_in, uint64_t d_out, uint32_t lora_rank);
int32_t strips_forward(const nf4_linear_args &a, cudaStream_t stream);
// T = x A in f32, [rows][rank], a CTA to a value: for few rows.  a: [d_in][r], or [r][d_in] (out_in)
int32_t small_lora_t(const void *x, const void *a, float *t, uint64_t rows, uint64_t K, uint32_t rank, bool f32, bool out_in, cudaStream_t stream);

// f32_rows.cu: f32 tensors, NF4_LAYOUT_OUT_IN, rows <= 16: rows split into bf16 halves for the decode kernels
bool f32_rows_supported(const nf4_linear_args &a);
uint64_t f32_rows_workspace_bytes(uint64_t rows, uint64_t d_in, uint64_t d_out, uint32_t lora_rank);
int32_t f32_rows_forward(const nf4_linear_args &a, cudaStream_t stream);

// prefill_gemm.cu: tcgen05 GEMM, NF4_LAYOUT_OUT_IN, bf16 activations.
bool prefill_supported(const nf4_linear_args &a);
// NF4_LAYOUT_IN_OUT at more than 16 rows, bf16 or f32 activations: repacked into the workspace, same GEMM
bool prefill_in_out_supported(const nf4_linear_args &a);
uint64_t prefill_workspace_bytes(uint64_t rows, uint64_t d_in, uint64_t d_out, uint32_t lora_rank);
int32_t prefill_code_place(uint32_t block, uint32_t *slot_full_parity);
int32_t prefill_share_plan(uint64_t rows, uint64_t d_in, uint64_t d_out, bool wide_only, uint32_t cta, uint32_t *tile_rows, uint32_t *ctas,
                           uint32_t *segments, uint32_t cap);
// r_out: null, or where x A goes too (see PrepassArgs)
int32_t prefill_forward(const nf4_linear_args &a, cudaStream_t stream, void *r_out = nullptr);

// prepass.cu: the f16 copy of the activations with its rows' factors, and the adapter intermediate.
// x [M][K] bf16 or f32 (K a multiple of 8, of 64 for f32, 16-byte aligned); a: the factor as [rank][K], or [K][rank]
// (k_major), of x's type.  xh null: r_out alone (bf16 x).  t_out and r_out: [M][2 * 64 * ceil(rank / 64)]
// bf16, hi halves then lo; t_out the scaled intermediate the GEMM adds, r_out (may be null) x a as it is.
// f32: r_out null, rank <= 128 and a multiple of four; t_out holds every column twice, as an adapter's of twice the rank.
struct PrepassArgs {
    const void *x;
    bool x_f32;
    uint32_t M, K;
    const void *a;
    uint32_t rank;
    bool k_major;
    float scale;
    void *xh;
    float *row_scale;
    void *t_out, *r_out;
    const float *absmax;
    const uint8_t *scale_codes;
    const float *scale_of_scales;
    uint32_t *flags;
    uint32_t n_flags;
};
int32_t activations_prepass(const PrepassArgs &q, cudaStream_t stream);

}  // namespace nf4
