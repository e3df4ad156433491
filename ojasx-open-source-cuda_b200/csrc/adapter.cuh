// Decode-shape linear of a layer with a low-rank adapter and, optionally, rotated weights:
//     y = H(x) . W^T (+ bias) + scaling * (x . A) . B
// as two launches: adapter_prologue_kernel (t = scaling * (x . A) in fp32, and H(x)) and the decode kernel, whose epilogue adds
// t . B.  Through the tensor library the same layer took a product of A (6.7 us at 4 x 4096 x 16), a conversion, a scaling, the
// transform and the decode kernel one after the other (23 us on the GPU and 77 us of host time per call); the two launches take
// 14.4 us, since the decode kernel starts beside the first and only waits for it before it reads x.
#pragma once

#include <cooperative_groups.h>

#include "fwht.cuh"
#include "gemv_host.cuh"

namespace ojx {

constexpr int kAdapterThreads = 512, kAdapterCluster = 8, kAdapterSlab = 16;     // a cluster sums 16 columns of A over all of K
constexpr int kAdapterMaxRank = 64;

// What bounds it: latency - 128 KB of A at the shape above.  Eight CTAs share K (16 KB of A each, two rounds of loads per thread)
// and add their sums through distributed shared memory; more CTAs would wait longer for each other than they save in loads.
// Grid: ceil(rank / 16) clusters for x . A, then, with rotated weights, one for the transform.
template <typename T, int MB>
__global__ void __launch_bounds__(kAdapterThreads, 1) __cluster_dims__(kAdapterCluster, 1, 1)
adapter_prologue_kernel(const T* __restrict__ x, const T* __restrict__ a, int M, int K, int rank, int vector_a, float scaling,
                        float* __restrict__ t_out, T* __restrict__ rot) {
    namespace cg = cooperative_groups;
    __shared__ float warp_sums[kAdapterThreads / 32][MB * kAdapterSlab];
    __shared__ float cta_sums[MB * kAdapterSlab];
    // the decode kernel may start: it reads nothing written here before this kernel has ended
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const int tid = threadIdx.x, lane = tid & 31, cta = (int)blockIdx.x % kAdapterCluster, slab = (int)blockIdx.x / kAdapterCluster;
    const int slabs = (rank + kAdapterSlab - 1) / kAdapterSlab;
    if (slab >= slabs) {                                            // the transform: a thread per block of 32
        const int64_t blocks = (int64_t)M * K / 32;
        for (int64_t b = (int64_t)tid * kAdapterCluster + cta; b < blocks; b += kAdapterThreads * kAdapterCluster) {
            const uint4* src = reinterpret_cast<const uint4*>(x + b * 32);
            uint4* dst = reinterpret_cast<uint4*>(rot + b * 32);
            uint32_t w[16];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint4 u = __ldg(src + c);
                w[c * 4 + 0] = u.x; w[c * 4 + 1] = u.y; w[c * 4 + 2] = u.z; w[c * 4 + 3] = u.w;
            }
            fwht32_pairs<T>(w);
#pragma unroll
            for (int c = 0; c < 4; ++c) dst[c] = make_uint4(w[c * 4 + 0], w[c * 4 + 1], w[c * 4 + 2], w[c * 4 + 3]);
        }
        return;                                                     // whole clusters take this branch
    }
    const int octet = tid & 1, col = slab * kAdapterSlab + octet * 8;
    const int k_end = (int)((int64_t)K * (cta + 1) / kAdapterCluster);
    cg::cluster_group cluster = cg::this_cluster();
    for (int m0 = 0; m0 < M; m0 += MB) {
        float acc[MB * 8];
#pragma unroll
        for (int i = 0; i < MB * 8; ++i) acc[i] = 0.f;
#pragma unroll (MB > 4 ? 1 : 2)
        for (int k = (int)((int64_t)K * cta / kAdapterCluster) + (tid >> 1); k < k_end; k += kAdapterThreads / 2) {
            float av[8];
            if (vector_a) {
                uint4 u = make_uint4(0, 0, 0, 0);
                if (col < rank) u = __ldg(reinterpret_cast<const uint4*>(a + (int64_t)k * rank + col));
                const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) { av[2 * i] = Pair16<T>::lo(w[i]); av[2 * i + 1] = Pair16<T>::hi(w[i]); }
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) av[i] = col + i < rank ? static_cast<float>(a[(int64_t)k * rank + col + i]) : 0.f;
            }
#pragma unroll
            for (int m = 0; m < MB; ++m) {
                if (m0 + m >= M) break;
                const float xv = static_cast<float>(x[(int64_t)(m0 + m) * K + k]);
#pragma unroll
                for (int i = 0; i < 8; ++i) acc[m * 8 + i] = fmaf(xv, av[i], acc[m * 8 + i]);
            }
        }
        // lanes with the same octet: halves of the sums change hands until each lane holds its share
        int n = MB * 8, at = 0;
#pragma unroll
        for (int o = 16; o >= 2; o >>= 1) {
            const bool up = (lane & o) != 0;
            if (n > 1) {
                n >>= 1;
#pragma unroll
                for (int i = 0; i < MB * 4; ++i) {
                    if (i >= n) break;
                    const float send = up ? acc[i] : acc[i + n], keep = up ? acc[i + n] : acc[i];
                    acc[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, o);
                }
                if (up) at += n;
            } else {
                acc[0] += __shfl_xor_sync(0xFFFFFFFFu, acc[0], o);
            }
        }
        // (with fewer sums than lanes several lanes hold the same one and store the same value)
#pragma unroll
        for (int i = 0; i < (MB * 8 + 15) / 16; ++i) {
            const int v = at + i;                                   // row v / 8, column v % 8 of this lane's octet
            warp_sums[tid >> 5][(v >> 3) * kAdapterSlab + octet * 8 + (v & 7)] = acc[i];
        }
        __syncthreads();
        for (int i = tid; i < MB * kAdapterSlab; i += kAdapterThreads) {
            float sum = 0.f;
#pragma unroll
            for (int w = 0; w < kAdapterThreads / 32; ++w) sum += warp_sums[w][i];
            cta_sums[i] = sum;
        }
        cluster.sync();
        for (int i = tid * kAdapterCluster + cta; i < MB * kAdapterSlab; i += kAdapterThreads * kAdapterCluster) {
            const int m = m0 + i / kAdapterSlab, c = slab * kAdapterSlab + i % kAdapterSlab;
            float sum = 0.f;
#pragma unroll
            for (int r = 0; r < kAdapterCluster; ++r) sum += cluster.map_shared_rank(cta_sums, r)[i];
            if (m < M && c < rank) t_out[(int64_t)m * rank + c] = scaling * sum;
        }
        cluster.sync();                                             // nobody leaves, or sums the next rows, while others read
    }
}

inline size_t adapter_round(size_t b) { return (b + 255) & ~(size_t)255; }

// 16-bit activations up to sixteen rows, as the decode kernels take them.
inline bool adapter_decode_ok(int fmt, int x_dtype, int64_t M, int64_t N, int64_t K, int group, int rank) {
    return (x_dtype == OJX_BF16 || x_dtype == OJX_F16) && rank > 0 && rank <= kAdapterMaxRank && gemv_mma_ok(fmt, M, N, K, group, x_dtype);
}

size_t linear_adapter_workspace_bytes_impl(int64_t M, int64_t K, int rank, int hadamard) {
    if (M <= 0 || M > 16 || K <= 0 || rank <= 0 || rank > kAdapterMaxRank) return 0;
    return adapter_round((size_t)M * rank * sizeof(float)) + (hadamard ? (size_t)M * K * 2 : 0);
}

template <typename T>
static int32_t adapter_prologue(const void* x, const void* a, int M, int K, int rank, float scaling, float* t, void* rot, cudaStream_t s) {
    const int grid = kAdapterCluster * ((rank + kAdapterSlab - 1) / kAdapterSlab + (rot ? 1 : 0));
    const int vector_a = rank % 8 == 0 && (reinterpret_cast<uintptr_t>(a) & 15) == 0;
    const T *xp = static_cast<const T*>(x), *ap = static_cast<const T*>(a);
    T* rp = static_cast<T*>(rot);
    if (M == 1) adapter_prologue_kernel<T, 1><<<grid, kAdapterThreads, 0, s>>>(xp, ap, M, K, rank, vector_a, scaling, t, rp);
    else if (M <= 2) adapter_prologue_kernel<T, 2><<<grid, kAdapterThreads, 0, s>>>(xp, ap, M, K, rank, vector_a, scaling, t, rp);
    else if (M <= 4) adapter_prologue_kernel<T, 4><<<grid, kAdapterThreads, 0, s>>>(xp, ap, M, K, rank, vector_a, scaling, t, rp);
    else adapter_prologue_kernel<T, 8><<<grid, kAdapterThreads, 0, s>>>(xp, ap, M, K, rank, vector_a, scaling, t, rp);
    return launch_status();
}

int32_t linear_adapter_impl(int fmt, const void* x, int x_dtype, int64_t M, const uint8_t* packed, const uint16_t* scales, const void* bias,
                            int64_t N, int64_t K, int group, const void* lora_a, const void* lora_b, int rank, float scaling, int hadamard,
                            void* y, int y_dtype, void* ws, size_t ws_bytes, cudaStream_t s) {
    OJX_RETURN_IF(fmt != 0 && fmt != 1 && fmt != 2, OJX_ERR_UNSUPPORTED);
    OJX_RETURN_IF(!x || !packed || !scales || !y || !lora_a || !lora_b || !ws, OJX_ERR_NULL);
    if (fmt == 0) group = effective_group(group);
    OJX_RETURN_IF(!adapter_decode_ok(fmt, x_dtype, M, N, K, group, rank), OJX_ERR_UNSUPPORTED);
    OJX_RETURN_IF(ws_bytes < linear_adapter_workspace_bytes_impl(M, K, rank, hadamard), OJX_ERR_WORKSPACE);
    OJX_RETURN_IF(((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(packed) | reinterpret_cast<uintptr_t>(scales) |
                    reinterpret_cast<uintptr_t>(ws)) & 15) != 0, OJX_ERR_UNSUPPORTED);
    OJX_RETURN_IF(check_arch() != OJX_OK, OJX_ERR_ARCH);
    float* t = static_cast<float*>(ws);
    void* rot = hadamard ? static_cast<uint8_t*>(ws) + adapter_round((size_t)M * rank * sizeof(float)) : nullptr;
    const int32_t st = x_dtype == OJX_BF16 ? adapter_prologue<__nv_bfloat16>(x, lora_a, (int)M, (int)K, rank, scaling, t, rot, s)
                                           : adapter_prologue<__half>(x, lora_a, (int)M, (int)K, rank, scaling, t, rot, s);
    OJX_RETURN_IF(st != OJX_OK, st);
    // the launch ahead is the prologue, which starts after everything before it has ended and writes no weights: the decode kernel
    // may fetch those at once
    const void* xr = rot ? rot : x;
    if (fmt == 0) return gemv_impl(xr, x_dtype, M, packed, scales, bias, N, K, group, y, y_dtype, nullptr, kNoScratch, s, t, lora_b, rank, 1);
    return linear_lowbit_impl(fmt, xr, x_dtype, M, packed, scales, bias, N, K, group, y, y_dtype, s, t, lora_b, rank, 1);
}

}  // namespace ojx
