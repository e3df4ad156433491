// Encoder and decoder of the 1.0-bit format: one byte per 8-block, the index of one of 256 vectors (the 240 roots of
// E8 and 16 axis vectors, all doubled: coordinates 0, +-1, +-2), weight = coordinate * scale with one fp16
// least-squares scale per group of g consecutive weights.
//
// Follows RootE8LatticePacker.pack / unpack (ojasx2/math/lattice.py:475-537).  The reference picks the code with
// argmax over torch.matmul(v, normalize(table)^T); on its CPU path every entry of that product is the chain
// acc = fma(v[k], t[k], acc), k = 0..7, from acc = 0, and the first maximum wins.  The same chains are evaluated
// here, sharing what the table's structure lets them share:
//   * two non-zeros +-c (c = fl(2 / sqrt 8)) at i < j:   fma(v[j], +-c, fl(v[i] * +-c))               112 codes
//   * (+-d)^8, even number of minus signs (d = c / 2):    a binary tree over the first seven signs, the eighth fixed by
//     parity; flipping all eight signs negates the chain exactly, so only the half with a leading minus is walked
//     and the other half is read off its minima                                                        128 codes
//   * one non-zero +-1 at i:                              -+v[i]                                        16 codes
// The scale is <w, q> / <q, q> with the sum in torch.sum's CPU order (chunks of eight into four vector accumulators in
// turn, accumulators added 0..3, lanes 0..7).
#pragma once

#include "codec.cuh"

namespace ojx {

struct RootBest {
    float val;
    int idx;
};

// Index of the best of the 256 table vectors for one 8-block of normalised weights.
__device__ __forceinline__ int root_argmax(const float (&v)[8]) {
    const float c = __uint_as_float(0x3f3504f3u);            // 0.70710677: 2 / fl(sqrt(8))
    const float d = __uint_as_float(0x3eb504f3u);            // 0.35355338: 1 / fl(sqrt(8))
    RootBest best;
    // --- 112 codes with two non-zeros: index = 4 * pair + 2 * (s1 > 0) + (s2 > 0), pairs (i, j) in lexicographic order
    {
        float p[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) p[i] = __fmul_rn(v[i], c);
        best.val = __fmaf_rn(v[1], -c, -p[0]);
        best.idx = 0;
        int idx = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = i + 1; j < 8; ++j)
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const float dot = __fmaf_rn(v[j], (s & 1) ? c : -c, (s & 2) ? p[i] : -p[i]);
                    if (dot > best.val) { best.val = dot; best.idx = idx; }
                    ++idx;
                }
    }
    // --- 128 codes (+-d)^8: bits b0..b6 of B choose the first seven signs (0 = minus), the eighth makes the number of
    // minus signs even; index = 112 + (B >> 1) over the 8-bit patterns in increasing order.  Walk b0 = 0 only.
    {
        float hi = 0.f, lo = 0.f;          // largest chain value (first occurrence) and smallest (last occurrence)
        int hi_at = -1, lo_at = -1;        // as 7-bit prefixes
        const float a0 = -__fmul_rn(v[0], d);
#pragma unroll
        for (int b = 0; b < 64; ++b) {     // bits b1..b6 of the pattern are bits 5..0 of b
            float acc = a0;
#pragma unroll
            for (int k = 1; k < 7; ++k) acc = __fmaf_rn(v[k], ((b >> (6 - k)) & 1) ? d : -d, acc);
            const int ones = __popc(b);                                   // plus signs among the first seven (b0 = 0)
            const bool last_plus = (ones & 1) != 0;                       // even number of minus signs over all eight
            acc = __fmaf_rn(v[7], last_plus ? d : -d, acc);
            if (hi_at < 0 || acc > hi) { hi = acc; hi_at = b; }
            if (lo_at < 0 || acc <= lo) { lo = acc; lo_at = b; }
        }
        // first half: pattern B = (0, b, last) -> index 112 + b; second half: the complement of (0, b, last) has
        // prefix 127 - b -> index 112 + 127 - b, value -acc; its first maximum is the LAST minimum of the first half
        if (hi > best.val) { best.val = hi; best.idx = 112 + hi_at; }
        if (-lo > best.val) { best.val = -lo; best.idx = 112 + 127 - lo_at; }
    }
    // --- 16 codes with one non-zero: index 240 + 2 i + (sign > 0), value -+v[i]
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        if (-v[i] > best.val) { best.val = -v[i]; best.idx = 240 + 2 * i; }
        if (v[i] > best.val) { best.val = v[i]; best.idx = 241 + 2 * i; }
    }
    return best.idx;
}

// Kept out of line for the pruned search: rare there, and its registers would halve the occupancy.
__device__ __noinline__ int root_argmax_walk(float v0, float v1, float v2, float v3, float v4, float v5, float v6, float v7) {
    const float v[8] = {v0, v1, v2, v3, v4, v5, v6, v7};
    return root_argmax(v);
}

// The same index without walking the 256 vectors.  Every chain is built from correctly rounded multiply-adds, which are
// monotone in each term, so the largest value of a class is reached by the signs of v itself:
//   * two non-zeros: 28 chains over |v|; the first pair that reaches the maximum;
//   * (+-d)^8: one chain over |v| when v has an even number of minus signs, else the best of the eight chains with one
//     sign flipped; patterns with two more flips are smaller by 2 d (|v_a| + |v_b|), which the roundings of a chain (below
//     2^-20 of its value) can only hide when two magnitudes are below 2^-17 of the sum - then the walk above decides, as it
//     does for NaN;
//   * one non-zero: the first largest magnitude.
// About 250 instructions instead of about 1000 per eight weights.
__device__ __forceinline__ int root_argmax_pruned(const float (&v)[8]) {
    const float c = __uint_as_float(0x3f3504f3u), d = __uint_as_float(0x3eb504f3u);
    float m[8], pre[8];
    uint32_t nat = 0;                                        // bit 7 - i: v[i] counts as plus
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        m[i] = fabsf(v[i]);
        pre[i] = i == 0 ? __fmul_rn(m[0], d) : __fmaf_rn(m[i], d, pre[i - 1]);
        nat |= (~__float_as_uint(v[i]) >> 31) << (7 - i);
    }
    const float tiny = pre[7] * 7.62939453125e-06f;          // 2^-17
    int small = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) small += m[i] > tiny ? 0 : 1;
    if (small >= 2) return root_argmax_walk(v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7]);

    // --- two non-zeros: the first row (i) and in it the first column (j) that reach the maximum
    float p[7], rowmax[7], big = 0.f;
#pragma unroll
    for (int i = 0; i < 7; ++i) {
        p[i] = __fmul_rn(m[i], c);
        rowmax[i] = __fmaf_rn(m[i + 1], c, p[i]);
#pragma unroll
        for (int j = i + 2; j < 8; ++j) rowmax[i] = fmaxf(rowmax[i], __fmaf_rn(m[j], c, p[i]));
        big = fmaxf(big, rowmax[i]);
    }
    int row = 0;
    float prow = p[0];
#pragma unroll
    for (int i = 6; i >= 1; --i)
        if (rowmax[i] == big) { row = i; prow = p[i]; }
    if (rowmax[0] == big) { row = 0; prow = p[0]; }
    int col = 7;
#pragma unroll
    for (int j = 7; j >= 1; --j)
        if (j > row && __fmaf_rn(m[j], c, prow) == big) col = j;
    float best = big;
    int idx = 4 * ((row * (15 - row)) / 2 + col - row - 1) + (int)(2 * ((nat >> (7 - row)) & 1u) + ((nat >> (7 - col)) & 1u));

    // --- (+-d)^8
    float vb = pre[7];
    uint32_t pat = nat;
    if (__popc(nat) & 1) {                                   // odd number of minus signs
        float ch[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            ch[k] = k == 0 ? -pre[0] : __fmaf_rn(m[k], -d, pre[k - 1]);
#pragma unroll
            for (int l = k + 1; l < 8; ++l) ch[k] = __fmaf_rn(m[l], d, ch[k]);
        }
        vb = ch[0];
#pragma unroll
        for (int k = 1; k < 8; ++k) vb = fmaxf(vb, ch[k]);
        pat = 0xFFFFu;
#pragma unroll
        for (int k = 0; k < 8; ++k)
            if (ch[k] == vb) pat = min(pat, nat ^ (1u << (7 - k)));      // the first of equal values
    }
    if (vb > best) { best = vb; idx = 112 + (int)(pat >> 1); }

    // --- one non-zero
    float top = m[0];
#pragma unroll
    for (int i = 1; i < 8; ++i) top = fmaxf(top, m[i]);
    if (top > best) {
        int at = 0;
#pragma unroll
        for (int i = 7; i >= 0; --i)
            if (m[i] == top) at = i;
        idx = 240 + 2 * at + (int)((nat >> (7 - at)) & 1u);
    }
    return idx;
}

// One thread per scale group.  GROUP 8 or 32 (0: any): the group's values are read again, 16 or 32 bytes at a time, for the
// sum of squares and for the codes - from L1 the second time - instead of being held in registers.
template <typename T, int GROUP>
__global__ void __launch_bounds__(128) encode1_kernel(const T* __restrict__ w, int64_t total, int group_rt, float sqrt_group,
                                                       uint8_t* __restrict__ packed, uint16_t* __restrict__ scales, int64_t ngroups) {
    const int group = GROUP > 0 ? GROUP : group_rt;
    for (int64_t gi = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; gi < ngroups; gi += (int64_t)gridDim.x * blockDim.x) {
        const int64_t base = gi * group;
        const bool vec = base + group <= total && (reinterpret_cast<uintptr_t>(w + base) & 15) == 0;
        auto load8 = [&](int b, float (&x)[8]) {
            if (vec) {
                const uint4* src = reinterpret_cast<const uint4*>(w + base + b * 8);
                constexpr int per = 16 / sizeof(T);
#pragma unroll
                for (int q = 0; q < 8 / per; ++q) {
                    const uint4 u = __ldg(src + q);
                    const T* e = reinterpret_cast<const T*>(&u);
#pragma unroll
                    for (int i = 0; i < per; ++i) x[q * per + i] = to_f32<T>(e[i]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) x[i] = base + b * 8 + i < total ? to_f32<T>(w[base + b * 8 + i]) : 0.f;
            }
        };
        float acc[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[j] = 0.f;
#pragma unroll
        for (int b = 0; b < group / 8; ++b) {
            float x[8];
            load8(b, x);
#pragma unroll
            for (int j = 0; j < 8; ++j)        // the square of a 16-bit float is exact in fp32: one fused operation rounds the same
                acc[j] = sizeof(T) == 2 ? __fmaf_rn(x[j], x[j], acc[j]) : __fadd_rn(acc[j], __fmul_rn(x[j], x[j]));
        }
        float s = acc[0];
#pragma unroll
        for (int j = 1; j < 8; ++j) s = __fadd_rn(s, acc[j]);
        const float scale = __fadd_rn(__fdiv_rn(__fsqrt_rn(s), sqrt_group), 1e-8f);
        const bool fast = scale >= 1e-7f && scale <= 1e30f;             // x / scale through the reciprocal, exactly (codec.cuh)
        const float rcp = fast ? __frcp_rn(scale) : 0.f;
        float dotacc[GROUP > 0 ? 1 : 4][8];                             // <w, q> in torch.sum's order; up to four blocks need one accumulator
#pragma unroll
        for (int u = 0; u < (GROUP > 0 ? 1 : 4); ++u)
#pragma unroll
            for (int j = 0; j < 8; ++j) dotacc[u][j] = 0.f;
        float qq = 0.f;                                                 // <q, q>: small integers, exact in any order
        uint8_t* out = packed + gi * (int64_t)(group / 8);
        uint32_t word = 0;
#pragma unroll 1
        for (int b = 0; b < group / 8; ++b) {
            float x[8], v[8];
            load8(b, x);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                if (fast) {
                    const float q0 = __fmul_rn(x[i], rcp);
                    v[i] = __fmaf_rn(__fmaf_rn(-scale, q0, x[i]), rcp, q0);
                } else {
                    v[i] = __fdiv_rn(x[i], scale);
                }
            }
            const int code = root_argmax_pruned(v);
            if (GROUP == 32) word |= (uint32_t)code << (8 * b);
            else out[b] = (uint8_t)code;
            const uint2 cw = __ldg(reinterpret_cast<const uint2*>(g_root_coords) + code);
            // coordinates -2..2 as floats: bytes 0..4 into the mantissa of 2^23, minus 2^23 + 2
            const uint32_t lo = ((cw.x & 0x7F7F7F7Fu) + 0x02020202u) ^ (cw.x & 0x80808080u), hi = ((cw.y & 0x7F7F7F7Fu) + 0x02020202u) ^ (cw.y & 0x80808080u);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float q = __uint_as_float(prmt(i < 4 ? lo : hi, 0x4B000000u, 0x7540u | (uint32_t)(i & 3))) - 8388610.0f;
                const float pr = __fmul_rn(x[i], q);
                qq = __fmaf_rn(q, q, qq);
                if (GROUP > 0) {
                    dotacc[0][i] = __fadd_rn(dotacc[0][i], pr);
                } else {
#pragma unroll
                    for (int u = 0; u < 4; ++u)
                        if ((b & 3) == u) dotacc[u][i] = __fadd_rn(dotacc[u][i], pr);
                }
            }
        }
        if (GROUP == 32) {
            if ((reinterpret_cast<uintptr_t>(out) & 3) == 0) *reinterpret_cast<uint32_t*>(out) = word;
            else
#pragma unroll
                for (int b = 0; b < 4; ++b) out[b] = (uint8_t)(word >> (8 * b));
        }
        float dot = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float lane = dotacc[0][j];
            if constexpr (GROUP == 0) lane = __fadd_rn(__fadd_rn(__fadd_rn(lane, dotacc[1][j]), dotacc[2][j]), dotacc[3][j]);
            dot = j == 0 ? lane : __fadd_rn(dot, lane);
        }
        scales[gi] = __half_as_ushort(__float2half_rn(__fdiv_rn(dot, fmaxf(qq, 1e-8f))));
    }
}

template <typename T>
static int32_t encode1_typed(const void* w, int64_t total, int group, uint8_t* packed, uint16_t* scales, cudaStream_t s) {
    const int64_t ngroups = (total + group - 1) / group;
    const float sg = (float)sqrt((double)group);
    int64_t blocks = (ngroups + 127) / 128;
    if (blocks > 148 * 64) blocks = 148 * 64;
    const T* wp = static_cast<const T*>(w);
    if (group == 8) encode1_kernel<T, 8><<<(unsigned)blocks, 128, 0, s>>>(wp, total, group, sg, packed, scales, ngroups);
    else if (group == 32) encode1_kernel<T, 32><<<(unsigned)blocks, 128, 0, s>>>(wp, total, group, sg, packed, scales, ngroups);
    else encode1_kernel<T, 0><<<(unsigned)blocks, 128, 0, s>>>(wp, total, group, sg, packed, scales, ngroups);
    return launch_status();
}

int32_t encode1_impl(const void* w, int w_dtype, int64_t rows, int64_t cols, int group, uint8_t* packed, uint16_t* scales,
                     cudaStream_t s) {
    OJX_RETURN_IF(!w || !packed || !scales, OJX_ERR_NULL);
    OJX_RETURN_IF(rows <= 0 || cols <= 0, OJX_ERR_SHAPE);
    OJX_RETURN_IF(check_arch() != OJX_OK, OJX_ERR_ARCH);
    if (group <= 0 || group % 8 != 0) group = 8;              // as the reference does (lattice.py:485-486)
    const int64_t total = rows * cols;
    switch (w_dtype) {
        case OJX_F32: return encode1_typed<float>(w, total, group, packed, scales, s);
        case OJX_F16: return encode1_typed<__half>(w, total, group, packed, scales, s);
        case OJX_BF16: return encode1_typed<__nv_bfloat16>(w, total, group, packed, scales, s);
        default: return OJX_ERR_DTYPE;
    }
}

// Decoder: one thread per 8 weights (one code byte, one scale), whose index is a shift for groups that are powers of two: the 64-bit
// division was what bounded it (14336 x 4096 to fp16: 42 -> 32 us).
template <typename T>
__global__ void __launch_bounds__(256) decode1_kernel(const uint8_t* __restrict__ packed, const uint16_t* __restrict__ scales,
                                                       int64_t total, int per_scale, int shift, T* __restrict__ out) {
    const int64_t chunks = (total + 7) / 8;
    for (int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; c < chunks; c += (int64_t)gridDim.x * blockDim.x) {
        const int code = packed[c];
        const uint32_t lo = g_root_coords[2 * code], hi = g_root_coords[2 * code + 1];
        const float sc = decode_scale<T>(scales[shift >= 0 ? c >> shift : c / per_scale]);
        alignas(16) T vals[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            vals[i] = from_f32<T>(__fmul_rn((float)(int)(int8_t)(((i < 4 ? lo : hi) >> (8 * (i & 3))) & 0xFFu), sc));
        T* dst = out + c * 8;
        if (c * 8 + 8 <= total && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
            for (int v = 0; v < (int)(8 * sizeof(T) / 16); ++v) reinterpret_cast<uint4*>(dst)[v] = reinterpret_cast<const uint4*>(vals)[v];
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (c * 8 + i < total) dst[i] = vals[i];
        }
    }
}

template <typename T>
static int32_t decode1_typed(const uint8_t* packed, const uint16_t* scales, int64_t total, int group, void* out, cudaStream_t s) {
    const int per_scale = group / 8;                                // groups are multiples of eight
    int shift = -1;                                                 // powers of two: no 64-bit division
    for (int b = 0; b < 28; ++b)
        if ((1 << b) == per_scale) shift = b;
    int64_t blocks = ((total + 7) / 8 + 255) / 256;
    if (blocks > 148 * 32) blocks = 148 * 32;
    decode1_kernel<T><<<(unsigned)blocks, 256, 0, s>>>(packed, scales, total, per_scale, shift, static_cast<T*>(out));
    return launch_status();
}

int32_t decode1_impl(const uint8_t* packed, const uint16_t* scales, int64_t rows, int64_t cols, int group, int out_dtype,
                     void* out, cudaStream_t s) {
    OJX_RETURN_IF(!packed || !scales || !out, OJX_ERR_NULL);
    OJX_RETURN_IF(rows <= 0 || cols <= 0 || group <= 0 || group % 8 != 0, OJX_ERR_SHAPE);
    OJX_RETURN_IF(check_arch() != OJX_OK, OJX_ERR_ARCH);
    const int64_t total = rows * cols;
    switch (out_dtype) {
        case OJX_F32: return decode1_typed<float>(packed, scales, total, group, out, s);
        case OJX_F16: return decode1_typed<__half>(packed, scales, total, group, out, s);
        case OJX_BF16: return decode1_typed<__nv_bfloat16>(packed, scales, total, group, out, s);
        default: return OJX_ERR_DTYPE;
    }
}

}  // namespace ojx
