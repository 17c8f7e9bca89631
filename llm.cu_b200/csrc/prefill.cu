// Row-batched kernels of the prompt phase, beside the tensor-core projections (gemm_tc.cu) and the block
// attention (attn_prefill.cu):
//
//   rmsnorm_rows   RMSNorm of M rows (replaces kernel_compute_rms_norm + kernel_compute_norm_tensor,
//                  inference.cu:272-375, for M rows at once): same partials of four elements, same
//                  binary reduction tree, eps added in double, IEEE division, FP16 rounding.
//   iota           positions pos0 .. pos0 + n - 1 for the embedding / RoPE-angle prologue.
#include "common.cuh"
#include "gemv_common.cuh"

namespace llmb {

constexpr int kNormThreads = 256;

__global__ void __launch_bounds__(kNormThreads)
rmsnorm_rows_kernel(const __half *__restrict__ x, const __half *__restrict__ gamma, __half *__restrict__ y, int d,
                    int n_pow2, double eps) {
    extern __shared__ float norm_part[];  // n_pow2 partials (d / 4 real ones, zero padded)
    __shared__ float rms_s;
    const int row = blockIdx.x, tid = threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();  // x is the previous kernel's output
    const uint4 *xr = reinterpret_cast<const uint4 *>(x + (size_t)row * d);
    const int nchunks = d >> 3;
    for (int c = tid; c < (n_pow2 >> 1); c += kNormThreads) {
        float p0 = 0.0f, p1 = 0.0f;
        if (c < nchunks) sumsq_partials(xr[c], p0, p1);
        norm_part[2 * c] = p0;
        norm_part[2 * c + 1] = p1;
    }
    __syncthreads();
    for (int off = n_pow2 >> 1; off >= 1; off >>= 1) {
        for (int t = tid; t < off; t += kNormThreads) norm_part[t] += norm_part[t + off];
        __syncthreads();
    }
    if (tid == 0) rms_s = sqrtf((float)(eps + (double)(norm_part[0] / (float)d)));
    __syncthreads();
    const float rms = rms_s;
    uint4 *yr = reinterpret_cast<uint4 *>(y + (size_t)row * d);
    const uint4 *gr = reinterpret_cast<const uint4 *>(gamma);
    for (int c = tid; c < nchunks; c += kNormThreads) yr[c] = rmsnorm_apply8(xr[c], __ldg(gr + c), rms);
}

__global__ void iota_kernel(int *dst, int first, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = first + i;
}

}  // namespace llmb

extern "C" int llmb_rmsnorm_rows(const uint16_t *d_x, const uint16_t *d_gamma, uint16_t *d_y, int m, int d, double eps,
                                 llmb_stream_t stream_) {
    using namespace llmb;
    if (!d_x || !d_gamma || !d_y || m <= 0 || d <= 0) return LLMB_ERR_INVALID;
    if ((d & 7) || (((uintptr_t)d_x | (uintptr_t)d_gamma | (uintptr_t)d_y) & 15)) {
        set_last_error("llmb_rmsnorm_rows: d must be a multiple of 8 and the pointers 16-byte aligned");
        return LLMB_ERR_UNSUPPORTED;
    }
    int n_pow2 = 2;
    while (n_pow2 < d / 4) n_pow2 <<= 1;
    if ((size_t)n_pow2 * 4 > 40 * 1024) {
        set_last_error("llmb_rmsnorm_rows: d above 40960 is not supported");
        return LLMB_ERR_UNSUPPORTED;
    }
    // launched with programmatic stream serialization: the kernel waits for its predecessor itself
    LLMB_CUDA_OK(launch_pdl(rmsnorm_rows_kernel, dim3(m), dim3(kNormThreads), (size_t)n_pow2 * 4, static_cast<cudaStream_t>(stream_),
                            true, reinterpret_cast<const __half *>(d_x), reinterpret_cast<const __half *>(d_gamma),
                            reinterpret_cast<__half *>(d_y), d, n_pow2, eps));
    return LLMB_OK;
}

extern "C" int llmb_iota_i32(int32_t *d_out, int first, int n, llmb_stream_t stream_) {
    using namespace llmb;
    if (!d_out || n <= 0) return LLMB_ERR_INVALID;
    iota_kernel<<<(n + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream_)>>>(d_out, first, n);
    LLMB_CUDA_OK(cudaGetLastError());
    return LLMB_OK;
}
