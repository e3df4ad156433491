// One entry for the packed linear of every format: which kernel serves a call is decided here, once, for the C ABI, the
// torch module (torch_glue.cpp) and the ctypes wrappers alike.
#pragma once

#include "gemv_host.cuh"
#include "gemm_tcgen05.cuh"

namespace ojx {

constexpr int kForceDecode = 1, kForceGemm = 2;        // flags of ojx_e8t_linear (tests)

// Batches of tokens run the tcgen05 kernel, up to sixteen rows the decode kernels: 28672 x 8192 at sixteen rows, 78 us against
// 106 us and more (whose smallest tile takes 35 us at K = 4096 whatever the token count).
// (2.0-bit weights are rounded to fp16 there, except where K is no multiple of 256: gemm_split.)  fp32 outputs with K no multiple of
// 256 came from the fp32 kernel, within 1e-7 to 3e-7 of the exact product (2-norm); that kernel's accumulators leave 3e-6 to 2e-5
// there, which 16-bit outputs do not show, so these stay on the decode kernels, 3e-7 to 5e-7 (linear_in_blocks).
inline bool linear_uses_gemm(int fmt, int x_dtype, int64_t M, int64_t N, int64_t K, int group, bool aligned, int y_dtype, int flags) {
    (void)N;
    if (flags & kForceDecode) return false;
    if (flags & kForceGemm) return true;               // the kernel's own checks report what it cannot take
    return M > 16 && (K % 256 == 0 || y_dtype != OJX_F32) && (x_dtype == OJX_BF16 || x_dtype == OJX_F16) && K % 32 == 0 && aligned &&
           (group == 32 || group == 16 || (fmt != 0 && group == 8));
}

inline int linear_group(int fmt, int group) { return fmt == 0 ? effective_group(group) : group; }

size_t linear_workspace_bytes_impl(int fmt, int x_dtype, int64_t M, int64_t N, int64_t K, int group, int flags) {
    group = linear_group(fmt, group);
    if (linear_uses_gemm(fmt, x_dtype, M, N, K, group, true, x_dtype, flags))
        return (x_dtype == OJX_BF16 || K % 256 != 0) ? gemm_fmt_workspace_bytes(fmt, M, N, K) : 256;
    return 0;
}

// Batches of tokens on a decode kernel, up to sixteen rows at a time (333 x 2912 -> 2000: 208 to 236 us; the scalar fp32 kernel 2950 to 3190).
static int32_t linear_in_blocks(int fmt, const void* x, int x_dtype, int64_t M, const uint8_t* packed, const uint16_t* scales, const void* bias,
                                int64_t N, int64_t K, int group, void* y, int y_dtype, cudaStream_t s) {
    const int64_t blocks = (M + 15) / 16;
    for (int64_t b = 0; b < blocks; ++b) {
        const int64_t m0 = M * b / blocks, m = M * (b + 1) / blocks - m0;
        const uint8_t* xb = static_cast<const uint8_t*>(x) + m0 * K * dtype_size(x_dtype);
        uint8_t* yb = static_cast<uint8_t*>(y) + m0 * N * dtype_size(y_dtype);
        const int32_t st = fmt == 0 ? gemv_impl(xb, x_dtype, m, packed, scales, bias, N, K, group, yb, y_dtype, nullptr, kNoScratch, s)
                                    : linear_lowbit_impl(fmt, xb, x_dtype, m, packed, scales, bias, N, K, group, yb, y_dtype, s, nullptr, nullptr, 0, 3);
        OJX_RETURN_IF(st != OJX_OK, st);
    }
    return OJX_OK;
}

int32_t linear_impl(int fmt, const void* x, int x_dtype, int64_t M, const uint8_t* packed, const uint16_t* scales,
                    const void* bias, int64_t N, int64_t K, int group, void* y, int y_dtype, void* ws, size_t ws_bytes,
                    int flags, cudaStream_t s) {
    OJX_RETURN_IF(fmt != 0 && fmt != 1 && fmt != 2, OJX_ERR_UNSUPPORTED);
    OJX_RETURN_IF((flags & ~(kForceDecode | kForceGemm)) != 0, OJX_ERR_UNSUPPORTED);
    group = linear_group(fmt, group);
    const bool aligned = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(packed) |
                           reinterpret_cast<uintptr_t>(scales)) & 15) == 0;
    if (linear_uses_gemm(fmt, x_dtype, M, N, K, group, aligned, y_dtype, flags))
        return gemm_fmt_impl(fmt, x, x_dtype, M, packed, scales, bias, N, K, group, y, y_dtype, ws, ws_bytes, s);
    if (M > 16 && !(flags & kForceDecode) && x && packed && scales && y && aligned && y_dtype == OJX_F32 && gemv_mma_ok(fmt, 16, N, K, group, x_dtype))
        return linear_in_blocks(fmt, x, x_dtype, M, packed, scales, bias, N, K, group, y, y_dtype, s);
    if (fmt == 0) return gemv_impl(x, x_dtype, M, packed, scales, bias, N, K, group, y, y_dtype, nullptr, kNoScratch, s);
    return linear_lowbit_impl(fmt, x, x_dtype, M, packed, scales, bias, N, K, group, y, y_dtype, s, nullptr, nullptr, 0, 3);
}

}  // namespace ojx
