// Decode-shape linear for 1..16 activation rows (bf16 or fp16) of every packed format on tensor cores (mma.sync, weights as
// the row operand):
//
//   y[m, n] = sum_k x[m, k] * W[n, k]  (+ bias, + low-rank term)        fp32 accumulation
//
// Replaces the reference's scalar fused kernels (ojasx2/math/csrc/ojasx_math_core.hpp:444,580-634) and, for small batches,
// _FusedE8GEMMFunction.forward (ojasx2/math/lattice.py:551-640).
//
// Weights enter the fp16 MMAs as EXACT fp16 values (sibling formats: for scales up to 32752; outputs over larger ones are computed
// again in fp32, mma_dense).  Ternary and 1.0-bit: coordinate * scale.  2.0-bit: (code - 2) * scale,
// which is exact where (code - 1.5) * scale is not; the missing 0.5 * scale per weight is 0.5 * sum over scale groups of
// scale * (sum of the group's x), one extra MMA per two scales of a lane whose A registers ARE the scale words and whose B
// registers hold the group sums as fp16 high and low parts.
//
// Work: a tile is 16 weight rows, an item up to two tiles x one chunk of K; K is cut into slices of 256 and chunks of at
// most 16 slices; warp w owns slice w of the chunk and keeps that slice of x in registers as MMA B fragments.  Every CTA owns
// a contiguous range of tiles and walks its items chunk-major.
//   * An item's rows travel by 16-byte cp.async (warp w copies rows w and w + 16) into a ring of stages with padded row
//     pitches, kDepth items ahead.  cp.async.bulk was measured and lost: rows whose address differs from their padded place
//     modulo 128 moved at 16 bytes per 4 cycles.  Rows of a matrix whose K is no multiple of 256 start at any even address:
//     they are copied with the bytes around them and read at their own offset (kRag).
//   * ONE barrier per item: it publishes the item's data and the previous item's partial sums and frees the previous stage.
//     Its threads then add the previous item up in warp order (deterministic).  K of several chunks keeps its running sums
//     in shared memory: no scratch in global memory and no second kernel.
//   * Lane (g, t) owns k 64t..64t+63 of the slice for rows g and g + 8 of a tile: eight 8-weight chunks, each two 64-bit
//     table reads (one 128-bit read for 1.0 bit), four packed multiplies by the scale and two MMAs per eight activation rows.
//     Table copies are interleaved so that no two lanes of an access meet in a bank.  A ternary rank r is the base-3 number
//     2r; its coordinates are the digits of (2r) mod 81 and (2r) div 81.
//   * x is read row by row (512 contiguous bytes) and brought into fragment order through shared memory: fetched directly, a
//     fragment load touches 32 cache lines, and sixteen rows cost every CTA 9 us before its first MMA.
#pragma once

#include <type_traits>

#include "gemv.cuh"

namespace ojx {

constexpr int kMmaWarps = 16;
constexpr int kMmaThreads = kMmaWarps * 32;
constexpr int kMmaAccTiles = 16;                     // tiles whose sums over K chunks are kept at a time
constexpr int kMmaXStageRows = 2;                    // up to so many activation rows travel inside the stages
constexpr int kMmaXRows = 2;                         // rows a warp brings into fragment order at a time
constexpr int kMmaXBytes = kMmaXRows * 512;          // its scratch for that

template <int FMT, int G>
struct MmaFmt {
    static constexpr int kCode = FMT == 0 ? 48 : (FMT == 2 ? 64 : 32);    // bytes of codes per row and slice
    static constexpr int kScale = 512 / G;                                 // bytes of scales per row and slice
    static constexpr int kCW = kCode / 16, kSW = kScale / 16;              // 32-bit words of a lane; also 16-byte vectors per row and slice
    static constexpr int kLut = FMT == 0 ? 104 * 128 : 256 * 128;          // rank 4095 (corrupt input) stays inside: 8190 div 81 = 101
    static constexpr int kBytes = kCode + kScale;
};

// Tiles of an item and items in flight.  Two tiles share the per-item work (barrier, copies, hand-over) where shared memory
// has room for their partial sums and stages: up to eight activation rows and 80 (kRag: 64) bytes per row and slice.
template <int FMT, int G, int NB, bool kRag>
struct MmaShape {
    static constexpr int kBytes = MmaFmt<FMT, G>::kBytes;
    static constexpr int kTiles = NB == 1 && kBytes <= (kRag ? 64 : 80) ? 2 : 1, kRows = 16 * kTiles;
    static constexpr int kDepth = kTiles == 2 ? (kBytes <= 48 ? 3 : 2) : (kBytes <= 64 ? 4 : (kBytes <= 96 ? 3 : 2));
    static constexpr int kStages = kDepth + 1;
    static constexpr int kPitch = kTiles == 2 ? 36 : 20;               // floats per activation row of a warp's partial sums: conflict-free stores
};

// Row pitch of `n` slices of `unit` bytes: the rows that one shared-memory access touches fall on distinct banks.
__host__ __device__ inline int mma_pitch(int n, int unit, bool rag) { return n * unit + ((n & 1) ? 0 : (unit == 48 ? 16 : unit)) + (rag ? 32 : 0); }

// Slices of 256 k, chunks of at most 16 slices, slices of a full chunk.
__host__ __device__ inline int mma_slices(int K) { return (K + 255) / 256; }
__host__ __device__ inline int mma_chunks(int K) { return (mma_slices(K) + kMmaWarps - 1) / kMmaWarps; }
__host__ __device__ inline int mma_per_chunk(int K) { const int c = mma_chunks(K); return (mma_slices(K) + c - 1) / c; }

struct MmaPlan {                                     // shared-memory layout, by the host
    int stage_bytes, scale_off, x_off;               // of a stage: scales, and x of a chunk's first item
    int x_staged;                                    // x travels inside the stages (up to kMmaXStageRows rows)
    int cluster;                                     // CTAs that share tiles and split the chunks of K
    int off_ring, off_part, off_acc, off_x, off_ctl; // byte offsets: ring, partial sums (two buffers), sums over chunks, x staging, control
    int total;
};

// Control block in shared memory.
struct MmaCtl {
    uint64_t never;                                  // tests: a barrier that nothing completes
    int abort_flag;
    ojx_e8t_gemv_problem prob;                       // the problem of a launch from a table
};

__device__ __forceinline__ uint2 lds_u64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts_f32(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
// 16-byte copy of which only `size` bytes are read, the rest written as zero.
__device__ __forceinline__ void cp_async16_part(uint32_t dst, const void* src, int size) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(size) : "memory");
}

// fp16 MMA with fp32 accumulation: D (16 x 8) += A (16 x 16, row-major) * B (16 x 8, column-major).
__device__ __forceinline__ void mma_f16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// the same with a zero accumulator operand: no registers to clear
__device__ __forceinline__ void mma_f16_zero(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
// int8 MMA with int32 accumulation: D (16 x 8) += A (16 x 32, row-major) * B (32 x 8, column-major).
__device__ __forceinline__ void mma_s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_s8_zero(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ uint32_t h2mul(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t pack_h2(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// N consecutive words at a shared-memory address of the given alignment.
template <int N, int ALIGN>
__device__ __forceinline__ void lds_words(uint32_t addr, uint32_t (&w)[N]) {
    if constexpr (ALIGN == 2) {
        const uint32_t a = addr & ~3u, sh = (addr & 2u) * 8u;
        uint32_t raw[N + 1];
#pragma unroll
        for (int i = 0; i <= N; ++i) raw[i] = lds_u32(a + 4 * i);
#pragma unroll
        for (int i = 0; i < N; ++i) w[i] = __funnelshift_r(raw[i], raw[i + 1], sh);
    } else if constexpr (N == 4 && ALIGN == 16) {
        const uint4 v = lds_u128(addr);
        w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    } else if constexpr (N == 2 && ALIGN >= 8) {
        const uint2 v = lds_u64(addr);
        w[0] = v.x; w[1] = v.y;
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i) w[i] = lds_u32(addr + 4 * i);
    }
}

// Bits [12 J, 12 J + 12) of a lane's 96-bit window, moved to start at bit 8 (bits outside the field are junk).
template <int J>
__device__ __forceinline__ uint32_t rank_at_8(const uint32_t (&w)[3]) {
    constexpr int bit = 12 * J, word = bit >> 5, off = bit & 31;
    if constexpr (off + 12 > 32) return __funnelshift_r(w[word], w[word + 1 < 3 ? word + 1 : 2], off - 8);
    else if constexpr (off > 8) return w[word] >> (off - 8);
    else return w[word] << (8 - off);
}

// Table reads: no `volatile`, so that the compiler may move them among the MMAs (their addresses come from the item's words).
template <int IMM> __device__ __forceinline__ uint32_t lut_u32(uint32_t at) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1+%2];" : "=r"(v) : "r"(at), "n"(IMM));
    return v;
}
template <int IMM> __device__ __forceinline__ uint2 lut_u64(uint32_t at) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2+%3];" : "=r"(v.x), "=r"(v.y) : "r"(at), "n"(IMM));
    return v;
}
template <int IMM> __device__ __forceinline__ uint4 lut_u128(uint32_t at) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4+%5];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at), "n"(IMM));
    return v;
}
// Table offsets of a ternary rank's low and high four digits, u = (2 rank) mod 81 and v = (2 rank) div 81, 128 bytes per entry.
// The field sits in the mantissa of F = 2 (1 + X 2^-23), X = 256 rank + the lane's offset; one multiply-add and one add round
// X / 20736 to v / 2 in the binade of 2^22, so the sum's bits are 0x4A800001 + v, and both offsets are one integer multiply-add
// of those bits (the constants cancel modulo 2^32).  Exact for every rank below 4096 and lane offset below 128 (checked
// exhaustively).  A multiply-high instead of the two float operations takes four cycles instead of two.
__device__ __forceinline__ void mma_digits(uint32_t field_at_8, uint32_t lane_f, uint32_t lane_v, uint32_t& u_at, uint32_t& v_at) {
    uint32_t f;
    asm("lop3.b32 %0, %1, 0xFFF00, %2, 0xEA;" : "=r"(f) : "r"(field_at_8), "r"(lane_f));          // (field & mask) | lane
    const float h = __fadd_rn(__fmaf_rn(__uint_as_float(f), __uint_as_float(0x434A4588u), __uint_as_float(0xC3CA6585u)), 4194304.5f);
    const uint32_t v = __float_as_uint(h);
    asm("mad.lo.u32 %0, %1, 4294956928, %2;" : "=r"(u_at) : "r"(v), "r"(f));                      // F - 10368 v: 10368 below the entry
    asm("mad.lo.u32 %0, %1, 128, %2;" : "=r"(v_at) : "r"(v), "r"(lane_v));
}
constexpr int kMmaDigitBias = 10368;
__device__ __forceinline__ uint32_t mma_lane_f(uint32_t offset) { return 0x40000000u | offset; }
__device__ __forceinline__ uint32_t mma_lane_v(uint32_t offset) { return offset - 0x40000000u - 128u; }

// Eight weights (chunk J of the lane's 64) as four fp16 pairs coordinate * scale.  `lut`: the table's address, `lane_at`: this lane's copy.
template <int FMT, int J, int CW>
__device__ __forceinline__ void mma_decode(uint32_t (&a)[4], const uint32_t (&w)[CW], uint32_t s2, uint32_t lut, uint32_t lane_at, uint32_t lane_f, uint32_t lane_v) {
    uint2 lo, hi;
    if constexpr (FMT == 0) {
        uint32_t u, v;
        mma_digits(rank_at_8<J>(w), lane_f, lane_v, u, v);
        lo = lut_u64<kMmaDigitBias>(u + lut);
        hi = lut_u64<0>(v);
    } else if constexpr (FMT == 2) {
        const uint32_t x = w[J >> 1];
        lo = lut_u64<0>((((J & 1) ? (x >> 9) : (x << 7)) & 0x7F80u) + lane_at);
        hi = lut_u64<0>((((J & 1) ? (x >> 17) : (x >> 1)) & 0x7F80u) + lane_at);
    } else {
        constexpr int sh = 8 * (J & 3) - 7;
        const uint32_t x = w[J >> 2];
        const uint4 q = lut_u128<0>(((sh < 0 ? x << (sh < 0 ? -sh : 0) : x >> (sh < 0 ? 0 : sh)) & 0x7F80u) + lane_at);
        lo = make_uint2(q.x, q.y);
        hi = make_uint2(q.z, q.w);
    }
    a[0] = h2mul(lo.x, s2); a[1] = h2mul(lo.y, s2); a[2] = h2mul(hi.x, s2); a[3] = h2mul(hi.y, s2);
}

// One output of a sibling format in plain fp32, for sums `sum` that came out as Inf or NaN, by whatever cause: scales above 32752,
// whose doubles ((code - 2) * scale, coordinates of +-2) fp16 does not have, and 2.0-bit products with Inf in x, where
// (code - 2) + 0.5 turns an infinity into NaN.  1.0-bit sums over other scales are the dense product's as they are.
template <int FMT>
__device__ __noinline__ float mma_dense(const ojx_e8t_gemv_problem& P, int group, int x_dtype, int m, int n, float sum) {
    const int64_t r0 = (int64_t)n * P.K;
    if (FMT == 1) {
        bool large = false;
        for (int i = 0; i < P.K / group; ++i) large = large || (P.scales[r0 / group + i] & 0x7FFFu) >= 0x7800u;
        if (!large) return sum;
    }
    float acc = 0.f;
    for (int k = 0; k < P.K; ++k) {
        const int64_t at = r0 + k;
        const float c = FMT == 2 ? (float)((P.packed[at >> 2] >> (2 * (int)(at & 3))) & 3) - 1.5f
                                 : (float)(int)(int8_t)((g_root_coords[2 * (int)P.packed[at >> 3] + (int)((at >> 2) & 1)] >> (8 * (int)(at & 3))) & 0xFFu);
        acc = fmaf(load_any(P.x, x_dtype, (int64_t)m * P.K + k), c * __half2float(__ushort_as_half(P.scales[at / group])), acc);
    }
    for (int r = 0; r < P.lora_rank; ++r) acc = fmaf(P.lora_t[m * P.lora_rank + r], load_any(P.lora_b, x_dtype, (int64_t)r * P.N + n), acc);
    return acc;
}
__device__ __forceinline__ float mma_load16(const void* p, bool f16, int64_t i) {
    const uint16_t v = __ldg(static_cast<const uint16_t*>(p) + i);
    return f16 ? __half2float(__ushort_as_half(v)) : __uint_as_float((uint32_t)v << 16);
}

// Inf / NaN activations of a slice (fed to the int8 MMAs as 0): lane r adds, in fp32, the products of weight row r of the item
// with them - Inf * 0 and anything * NaN give NaN, as in fp32 arithmetic.
__device__ __noinline__ void mma_add_non_finite(const void* x, int slice, const uint8_t* codes, const uint16_t* scl, float* sum) {
    const int lane = threadIdx.x & 31;
    const uint4 q = __ldcg(reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(x) + (int64_t)slice * 256 + lane * 8));
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
    bool mine = false;
#pragma unroll
    for (int i = 0; i < 4; ++i) mine = mine || ((w[i] << 16) & 0x7FFFFFFFu) >= 0x7F800000u || (w[i] & 0x7FFF0000u) >= 0x7F800000u;
    uint32_t holders = __ballot_sync(0xFFFFFFFFu, mine);
    float corr = 0.f;
    while (holders != 0u) {
        const int l = __ffs(holders) - 1;                      // rank l of the slice = the eight values lane l holds
        holders &= holders - 1u;
        uint32_t xv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) xv[i] = __shfl_sync(0xFFFFFFFFu, w[i], l);
        const uint32_t b0 = codes[(3 * l) >> 1], b1 = codes[((3 * l) >> 1) + 1];
        const uint32_t rank = (l & 1) ? ((b0 >> 4) | (b1 << 4)) : (b0 | ((b1 & 0xFu) << 8));
        const uint32_t entry = g_trit_nibbles[rank < (uint32_t)kNumPoints ? rank : 0u];
        const float sc = __half2float(__ushort_as_half(scl[l >> 2]));
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint32_t bits = (i & 1) ? (xv[i >> 1] & 0xFFFF0000u) : (xv[i >> 1] << 16);
            if ((bits & 0x7FFFFFFFu) >= 0x7F800000u) {
                const uint32_t sel = (entry >> (4 * i)) & 0xFu;
                const float coord = sel == 1u ? 1.f : (sel == 2u ? -1.f : 0.f);
                corr += (coord * sc) * __uint_as_float(bits);
            }
        }
    }
    __syncwarp();                                              // the lanes' own partial sums are written
    *sum += corr;
}

// Threads of a warp may arrive one by one (their code before it branches), so not the .aligned form.
__device__ __forceinline__ void mma_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
}
// A float of CTA `rank`'s shared memory, at this CTA's address.
__device__ __forceinline__ float mma_ld_cluster(uint32_t addr, int rank) {
    uint32_t a;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

// The other ranks' copies of an output per lane, by all lanes of a warp: 8 << qs neighbouring lanes hold eight consecutive weight rows,
// each row's value in the first of its 1 << qs lanes (`out`: that lane has one).  Eight 16-bit outputs leave as one 16-byte vector per
// rank, a lane of the group each, instead of eight 2-byte stores (eight windows, here on one GPU, 4096 x 4096: 7.4 -> 6.6 us at one row,
// 15.5 -> 13.6 at sixteen; two windows 6.4 and 13.6 either way).
__device__ __noinline__ void mma_store_peers(const PeerMap& pm, void* y, int y_dtype, int64_t ld, int col, int n, int qs, bool out, float v) {
    const int lane = threadIdx.x & 31, base = lane & -(8 << qs);
    const uint32_t h = y_dtype == OJX_BF16 ? __bfloat16_as_ushort(__float2bfloat16_rn(v)) : __half_as_ushort(__float2half_rn(v));
    const uint32_t rows = qs == 0 ? 0xFFu : (qs == 1 ? 0x5555u : 0x11111111u);
    const bool whole = ((__ballot_sync(0xFFFFFFFFu, out) >> base) & rows) == rows;
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
        w[i] = __shfl_sync(0xFFFFFFFFu, h, base + ((2 * i) << qs)) | (__shfl_sync(0xFFFFFFFFu, h, base + ((2 * i + 1) << qs)) << 16);
    if (whole && pm.wide && y_dtype != OJX_F32 && (ld & 7) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0) {
        const int r = lane - base;
        if (r < pm.world && pm.delta[r] != 0)
            *reinterpret_cast<uint4*>(static_cast<uint8_t*>(y) + pm.delta[r] + (col * ld + (n & ~7)) * 2) = make_uint4(w[0], w[1], w[2], w[3]);
    } else if (out) {
        store_peers(pm, y, y_dtype, col * ld + n, v);
    }
}

// Decode table in shared memory, entry stride 128 bytes: sixteen 8-byte copies (1.0 bit: eight of 16 bytes, int8: 32 of 4
// bytes), so that every lane of an access reads banks of its own.  Four threads per entry, two 16-byte stores each.
template <int FMT, bool kI8>
__device__ __forceinline__ void mma_fill_table(uint8_t* smem, int tid) {
    constexpr int kEntries = FMT == 0 ? 104 : 256;
#pragma unroll
    for (int e0 = 0; e0 < kEntries; e0 += kMmaThreads / 4) {
        const int entry = e0 + (tid >> 2);
        if (entry >= kEntries) break;
        uint4 v;
        if constexpr (FMT == 0) {                              // four base-3 digits, each minus one (entries from 81 on: corrupt input, zero)
            uint32_t e = (uint32_t)entry, h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t q = (e * 171u) >> 9, d = e - 3u * q;                     // e div 3, exact below 256
                h[k] = entry >= 81 || d == 1u ? 0u : (d == 0u ? 0xBC00u : 0x3C00u);
                e = q;
            }
            if constexpr (kI8) {
                uint32_t w = 0u;
#pragma unroll
                for (int k = 0; k < 4; ++k) w |= (h[k] == 0u ? 0u : (h[k] == 0x3C00u ? 1u : 0xFFu)) << (8 * k);
                v = make_uint4(w, w, w, w);
            } else {
                v = make_uint4(h[0] | (h[1] << 16), h[2] | (h[3] << 16), h[0] | (h[1] << 16), h[2] | (h[3] << 16));
            }
        } else if constexpr (FMT == 2) {                       // a byte of codes -> four values code - 2
            constexpr uint32_t lo = 0xBC00C000u, hi = 0x3C000000u;
            uint32_t h[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) { const int c = (entry >> (2 * k)) & 3; h[k] = ((c & 2 ? hi : lo) >> (16 * (c & 1))) & 0xFFFFu; }
            v = make_uint4(h[0] | (h[1] << 16), h[2] | (h[3] << 16), h[0] | (h[1] << 16), h[2] | (h[3] << 16));
        } else {
            const uint32_t cw[2] = {g_root_coords[2 * entry], g_root_coords[2 * entry + 1]};
            uint32_t h[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                const int c = (int)(int8_t)((cw[k >> 2] >> (8 * (k & 3))) & 0xFFu);
                h[k] = c == 0 ? 0u : (c == 1 ? 0x3C00u : (c == -1 ? 0xBC00u : (c == 2 ? 0x4000u : 0xC000u)));
            }
            v = make_uint4(h[0] | (h[1] << 16), h[2] | (h[3] << 16), h[4] | (h[5] << 16), h[6] | (h[7] << 16));
        }
        uint4* dst = reinterpret_cast<uint4*>(smem + entry * 128 + (tid & 3) * 32);
        dst[0] = v;
        dst[1] = v;
    }
}

// One matrix: the problem is the kernel parameter, or (kGroup) the entry of a grouped launch's table in device memory.
//
// kI8: one bf16 activation row of ternary codes with groups of 32 on int8 MMAs (m16n8k32).  The table holds four coordinates
// per 32-bit entry, 32 copies: two conflict-free reads ARE the two operand registers of a rank - half the wavefronts of the
// fp16 form and no multiplies.  x is fixed point per scale group: the group's largest finite magnitude fixes an exponent E,
// q = rint(x 2^(26 - E)), |q| <= 2^27, in four balanced base-128 digits; values within 2^-19 of the group's maximum are exact,
// smaller ones are rounded at 2^-27 of it.  Accumulator column 2t' + h takes digits 2h, 2h + 1 of the group that lane quarter t'
// decodes, so only lane (g, t) with g >> 1 == t feeds column g; a group's integer sums are put together and scaled once.
// Inf / NaN enter the MMAs as 0 and are added back in fp32.
template <int FMT, int G, int NB, bool kRag, bool kGroup, bool kI8 = false>
__global__ void __launch_bounds__(kMmaThreads, 1)
gemv_mma_kernel(const ojx_e8t_gemv_problem* __restrict__ probs, const __grid_constant__ ojx_e8t_gemv_problem single,
                int M, int x_dtype, int y_dtype, int overlap, const __grid_constant__ MmaPlan plan,
                const __grid_constant__ PeerMap peers) {
    static_assert(!kI8 || (FMT == 0 && G == 32 && NB == 1 && !kRag), "the int8 form serves one bf16 row of ternary codes");
    using F = MmaFmt<FMT, G>;
    using Sh = MmaShape<FMT, G, NB, kRag>;
    constexpr int S = Sh::kStages, D = Sh::kDepth, T = Sh::kTiles, R = Sh::kRows;
    if constexpr (kI8) { M = 1; x_dtype = OJX_BF16; }                    // known, so that nothing below keeps registers for them
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t base = smem_u32(smem);                                // in a cluster: with this CTA's rank in its upper bits
    MmaCtl* ctl = reinterpret_cast<MmaCtl*>(smem + plan.off_ctl);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;

    // the launch that follows in the stream may start its own set-up now
    if (overlap) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (tid == 0) ctl->abort_flag = 0;
    // this lane's copy of the table
    const uint32_t lane_off = kI8 ? lane * 4 : (FMT == 1 ? (lane & 7) * 16 : (lane & 15) * 8);
    const uint32_t lane_at = lane_off + base, lane_f = mma_lane_f(lane_off), lane_v = mma_lane_v(lane_at);
    // A launch whose weights were not promised static waits for the kernel ahead before it reads anything; its table is ready by
    // then.  A static launch starts its copies first and fills the table while they travel.
    if (!kGroup) mma_fill_table<FMT, kI8>(smem, tid);
    if (overlap == 3) asm volatile("griddepcontrol.wait;" ::: "memory");

    // the CTAs of a cluster work on the same tiles, CTA `cr` on chunks cr, cr + cs, ... of K
    const int cs = plan.cluster, cr = (int)blockIdx.x % cs;
    const int K = kGroup ? probs->K : single.K, N = kGroup ? probs->N : single.N;
    // an even share of the tiles
    const int64_t tiles = (N + 15) / 16;
    const int t0 = (int)(tiles * (blockIdx.x / cs) / (gridDim.x / cs)), t1 = (int)(tiles * (blockIdx.x / cs + 1) / (gridDim.x / cs));
    const bool signal = peers.sync != nullptr && (peers.mode & OJX_GEMV_SIGNAL_PEERS) != 0;

    uint32_t xb[NB][8][4];                      // B fragments: [block][8-weight chunk j][k 0-1, 2-3, 4-5, 6-7 of the chunk]; kI8: [j][digit pair m, k half r] at [2 m + r]
    uint32_t xc[NB][F::kSW][2];                 // 2.0-bit: half the scale groups' sums of x, high and low parts, two groups each
    float up[NB][2];                            // 2^e of activation rows 2t, 2t + 1 of the block (this lane's output columns); kI8: of its two groups
    float upb[2] = {1.f, 1.f};                  // kI8: second factor
    bool xbad = false;                          // kI8: the warp's slice holds Inf or NaN
    const bool xf16 = x_dtype == OJX_F16;
    const int slot = M * (Sh::kPitch * 4);    // bytes of a warp's partial sums of an item: [column][kPitch] floats
    const uint32_t part = base + plan.off_part;
    float* acc_sums = reinterpret_cast<float*>(smem + plan.off_acc);
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
#pragma unroll
        for (int j = 0; j < 8; ++j) xb[nb][j][0] = xb[nb][j][1] = xb[nb][j][2] = xb[nb][j][3] = 0u;
#pragma unroll
        for (int i = 0; i < F::kSW; ++i) xc[nb][i][0] = xc[nb][i][1] = 0u;
        up[nb][0] = up[nb][1] = 1.0f;
    }
    bool col_on[NB][2];
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) { col_on[nb][0] = nb * 8 + 2 * t < M; col_on[nb][1] = nb * 8 + 2 * t + 1 < M; }
    // sums over the warps: 2^qs threads per (weight row, activation row)
    int qs = 0;
    while (qs < 2 && ((R * M) << (qs + 1)) <= kMmaThreads) ++qs;
    const int q_row = (tid >> qs) % R, q_col = (tid >> qs) / R, q_sub = tid & ((1 << qs) - 1), q_per = kMmaWarps >> qs;
    const bool x_staged = plan.x_staged != 0;

    bool first_run = true, dead = false;
    int stage = 0, buf = 0;
    auto code_bytes = [](uint32_t k) { return FMT == 0 ? k / 16 * 3 : (FMT == 2 ? k / 4 : k / 8); };       // k: multiples of 32

    {
        // of a table's entry, what the loader needs is kept in registers, the rest (read after the next barrier) in shared memory
        const ojx_e8t_gemv_problem& P = kGroup ? ctl->prob : single;
        const ojx_e8t_gemv_problem& P0 = kGroup ? *probs : single;
        const uint8_t* const codes = P0.packed;
        const uint8_t* const scales = reinterpret_cast<const uint8_t*>(P0.scales);
        const void* const x = P0.x;
        if (kGroup && tid < (int)(sizeof(ojx_e8t_gemv_problem) / 8))
            reinterpret_cast<uint64_t*>(&ctl->prob)[tid] = reinterpret_cast<const uint64_t*>(probs)[tid];
        const int slices = mma_slices(K), chunks = mma_chunks(K), per = mma_per_chunk(K);
        const int pc = mma_pitch(per, F::kCode, kRag), ps = mma_pitch(per, F::kScale, kRag);
        const uint32_t rc = code_bytes(K), rs = (uint32_t)K / G * 2;
        // blocks of tiles: all of them when K is one chunk, else as many as there is room for running sums; chunk-major inside
        for (int b0 = t0; b0 < t1; b0 += kMmaAccTiles) {
            const int nt = chunks == 1 ? t1 - b0 : min(kMmaAccTiles, t1 - b0), np = (nt + T - 1) / T;
            const int total = chunks > cr ? np * ((chunks - cr + cs - 1) / cs) : 0;

            // ---- loader: warp w copies rows w and w + 16 of an item, 16-byte vector lane, lane + 32, ... of the codes and then of
            // the scales.  Between items only the two row offsets are kept (bytes; the host keeps both buffers below 4 GB): registers
            // are what the decoder lacks. ----
            constexpr int NV = (F::kBytes + 31) / 32 + (kRag ? 1 : 0);             // vectors per lane and row at sixteen slices
            uint32_t l_c = 0, l_s = 0;                                              // this warp's row in the item's first tile
            int l_pair = 0, l_chunk = cr, istage = stage;
            auto copy_x = [&](int chunk, uint32_t st) {                            // this warp's slice of x, row by row
                const int k = (chunk * per + warp) * 256 + lane * 8;
                if (warp < min(per, slices - chunk * per)) {
                    const uint16_t* xp = static_cast<const uint16_t*>(x) + (k < K ? k : 0);
#pragma unroll
                    for (int r = 0; r < kMmaXStageRows; ++r)
                        if (r < M)
                            cp_async16_part(st + plan.x_off + (warp * M + r) * 512 + (lane ^ ((2 * (lane >> 3) + r) & 7)) * 16, xp + (int64_t)r * K, k < K ? 16 : 0);
                }
            };
            auto issue = [&](int n, bool with_x) {                                 // one commit group per call, also when nothing is left
                if (n < total) {
                    const uint32_t st = base + plan.off_ring + istage * plan.stage_bytes;
                    const int k0 = l_chunk * per * 256, k1 = min(K, k0 + min(per, slices - l_chunk * per) * 256);
                    if (l_pair == 0) {
                        l_c = (uint32_t)(b0 * 16 + warp) * rc + code_bytes(k0);
                        l_s = (uint32_t)(b0 * 16 + warp) * rs + (uint32_t)k0 / G * 2;
                    }
                    const uint32_t cn = code_bytes(k1) - code_bytes(k0), sn = (uint32_t)(k1 - k0) / G * 2;
#pragma unroll
                    for (int tt = 0; tt < T; ++tt) {
                        const int tile = l_pair * T + tt;
                        if (tile < nt && (b0 + tile) * 16 + warp < N) {
                            const uint32_t c0 = l_c & (kRag ? ~15u : ~0u), s0 = l_s & (kRag ? ~15u : ~0u);
                            const int nc = (int)((l_c + cn - c0 + 15) >> 4), ns = (int)((l_s + sn - s0 + 15) >> 4);
                            const uint32_t cd = st + (tt * 16 + warp) * pc, sd = st + plan.scale_off + (tt * 16 + warp) * ps;
#pragma unroll (NV > 3 ? 1 : NV)
                            for (int v = 0; v < NV; ++v) {
                                const int at = lane + 32 * v;
                                const bool code = at < nc;
                                const uint32_t b = (uint32_t)(code ? at : at - nc) * 16, from = (code ? c0 : s0) + b;
                                const uint8_t* src = (code ? codes : scales) + from;
                                if constexpr (kRag) {                              // never past the end of the buffer
                                    const uint32_t end = (uint32_t)N * (code ? rc : rs);
                                    if (at < nc + ns && from < end) cp_async16_part((code ? cd : sd) + b, src, (int)min(16u, end - from));
                                } else {
                                    if (at < nc + ns) cp_async16((code ? cd : sd) + b, src);
                                }
                            }
                        }
                        l_c += 16 * rc;
                        l_s += 16 * rs;
                    }
                    if (with_x && l_pair == 0 && x_staged) copy_x(l_chunk, st);
                    if (++l_pair == np) { l_pair = 0; l_chunk += cs; }
                    if (++istage == S) istage = 0;
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            };
            // packed weights of a static launch do not depend on the launch ahead: their copies start before it has drained
            for (int i = 0; i < D; ++i) issue(i, !(first_run && overlap == 1));
            if (first_run) {
                if (kGroup) mma_fill_table<FMT, kI8>(smem, tid);
                // activations (and the output buffers) depend on the launch ahead, unless the caller declared this one independent
                if (overlap == 1) asm volatile("griddepcontrol.wait;" ::: "memory");
                // ... and, in a column-sharded chain, on the same launch of every other rank
                if (peers.sync != nullptr && (peers.mode & OJX_GEMV_WAIT_PEERS)) {
                    if (tid == 0) peer_wait(peers);
                    __syncthreads();
                }
                if (overlap == 1 && x_staged) {
                    for (int i = 0; i < D && i < total; ++i)
                        if (i % np == 0) copy_x(cr + i / np * cs, base + plan.off_ring + i * plan.stage_bytes);
                    asm volatile("cp.async.wait_all;" ::: "memory");
                }
                if (peers.lose_copy) {                                              // tests: a wait that runs out
                    if (tid == 0) { mbar_init(smem_u32(&ctl->never), 1); asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
                    __syncthreads();
                    dead = !mbar_wait(smem_u32(&ctl->never), 0u, &ctl->abort_flag, 52, peers.wait_limit);
                    dead = __syncthreads_or(dead);
                }
            }

            // ---- x of a chunk into B fragments; registers of lanes that feed no column stay zero from the start ----
            auto load_x = [&](int chunk, uint32_t st) {
                const int slice = chunk * per + warp;
                const bool active = warp < min(per, slices - chunk * per);
                const uint32_t xs = base + plan.off_x + warp * kMmaXBytes;
                if constexpr (kI8) {
                    // four lanes share a scale group
                    const uint4 q = active ? lds_u128(st + plan.x_off + warp * 512 + (lane ^ ((2 * (lane >> 3)) & 7)) * 16) : make_uint4(0, 0, 0, 0);
                    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
                    uint32_t m2 = __vmaxu2(__vmaxu2(w[0] & 0x7FFF7FFFu, w[1] & 0x7FFF7FFFu), __vmaxu2(w[2] & 0x7FFF7FFFu, w[3] & 0x7FFF7FFFu));
                    uint32_t amax = max(m2 & 0xFFFFu, m2 >> 16);                            // bf16 bits of the largest magnitude
                    const bool bad = amax >= 0x7F80u;
                    if (__any_sync(0xFFFFFFFFu, bad)) {
                        // rare: the largest FINITE magnitude of the group, and Inf / NaN as 0
                        xbad = true;
                        amax = 0;
#pragma unroll
                        for (int i = 0; i < 8; ++i) { const uint32_t mag = (i & 1 ? w[i >> 1] >> 16 : w[i >> 1]) & 0x7FFFu; if (mag < 0x7F80u) amax = max(amax, mag); }
                    } else {
                        xbad = false;
                    }
                    amax = max(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
                    amax = max(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 2));
                    const int ex = (int)(amax >> 7);
                    const int shift = 26 - (ex == 0 ? -126 : ex - 127);                     // in [-101, 152]: 2^shift applied as two factors
                    const int fa_e = shift >> 1, fb_e = shift - fa_e;
                    const float fa = __uint_as_float((uint32_t)(127 + fa_e) << 23), fb = __uint_as_float((uint32_t)(127 + fb_e) << 23);
                    uint32_t dw[4][2];                                                      // [digit][values 0-3, 4-7] as int8 x 4
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        uint32_t s[4];                                                      // a value's digits in four bytes: signed top, then 7 bits each
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            const int i = 4 * h + j;
                            uint32_t vb = (i & 1) ? (w[i >> 1] & 0xFFFF0000u) : (w[i >> 1] << 16);
                            if (xbad && (vb & 0x7FFFFFFFu) >= 0x7F800000u) vb = 0u;
                            uint32_t q0 = (uint32_t)__float2int_rn(__uint_as_float(vb) * fa * fb);
                            q0 += q0 & 0xFFFFFF80u;                                         // everything above the lowest digit moves up one bit, and so on
                            q0 += q0 & 0xFFFF8000u;
                            s[j] = q0 + (q0 & 0xFF800000u);
                        }
                        const uint32_t a = prmt(s[0], s[1], 0x5140u), b = prmt(s[2], s[3], 0x5140u);     // bytes 0, 1 of two values each
                        const uint32_t c = prmt(s[0], s[1], 0x7362u), d = prmt(s[2], s[3], 0x7362u);     // bytes 2, 3
                        dw[3][h] = prmt(a, b, 0x5410u); dw[2][h] = prmt(a, b, 0x7632u);
                        dw[1][h] = prmt(c, d, 0x5410u); dw[0][h] = prmt(c, d, 0x7632u);
                    }
                    // cell (digit pair h, lane l) is 16 bytes at slot l ^ (2 (l >> 3)) of half h
                    const uint32_t cell = xs + (lane ^ ((2 * (lane >> 3)) & 7)) * 16;
                    __syncwarp();
                    sts_u128(cell, make_uint4(dw[0][0], dw[0][1], dw[1][0], dw[1][1]));
                    sts_u128(cell + 512, make_uint4(dw[2][0], dw[2][1], dw[3][0], dw[3][1]));
                    __syncwarp();
                    if ((g >> 1) == t) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const uint4 v = lds_u128(xs + (g & 1) * 512 + (8 * t + (j ^ (2 * t))) * 16);
                            xb[0][j][0] = v.x; xb[0][j][1] = v.y; xb[0][j][2] = v.z; xb[0][j][3] = v.w;
                        }
                    }
                    const float una = __uint_as_float((uint32_t)(127 - fa_e) << 23), unb = __uint_as_float((uint32_t)(127 - fb_e) << 23);
                    up[0][0] = __shfl_sync(0xFFFFFFFFu, una, 8 * t);     upb[0] = __shfl_sync(0xFFFFFFFFu, unb, 8 * t);       // group 2t
                    up[0][1] = __shfl_sync(0xFFFFFFFFu, una, 8 * t + 4); upb[1] = __shfl_sync(0xFFFFFFFFu, unb, 8 * t + 4);   // group 2t + 1
                } else {
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) {
                        if (x_staged) {                                       // rows lie in the stage, 512 bytes each, vectors of row r at slot v ^ (2 (v >> 3) + r)
                            if (active && nb == 0 && g < M) {
#pragma unroll
                                for (int j = 0; j < 8; ++j) {
                                    const uint4 v = lds_u128(st + plan.x_off + (warp * M + g) * 512 + (8 * t + (j ^ ((2 * t + g) & 7))) * 16);
                                    xb[nb][j][0] = v.x; xb[nb][j][1] = v.y; xb[nb][j][2] = v.z; xb[nb][j][3] = v.w;
                                }
                            }
                        } else {
                            const bool mine = active && (!kRag || slice * 256 + lane * 8 < K);
                            const uint4* xrow = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(x) + (int64_t)slice * 256) + lane;
                            const int64_t pitch = K / 8;
                            uint4 raw[8];                                     // rows nb * 8 ..: this lane's eight k of each
#pragma unroll
                            for (int r = 0; r < 8; ++r) {
                                raw[r] = make_uint4(0, 0, 0, 0);
                                if (mine && nb * 8 + r < M) raw[r] = __ldcg(xrow + (nb * 8 + r) * pitch);   // L2: in a sharded chain x was written by other GPUs
                            }
#pragma unroll
                            for (int q = 0; q < 4; ++q) {                     // two rows at a time
                                if (nb * 8 + 2 * q >= M) break;
                                __syncwarp();
#pragma unroll
                                for (int r = 0; r < 2; ++r)
                                    sts_u128(xs + r * 512 + (lane ^ ((2 * (lane >> 3) + r) & 7)) * 16, raw[2 * q + r]);
                                __syncwarp();
                                if ((g >> 1) == q) {
#pragma unroll
                                    for (int j = 0; j < 8; ++j) {
                                        const uint4 v = lds_u128(xs + (g & 1) * 512 + (8 * t + (j ^ ((2 * t + (g & 1)) & 7))) * 16);
                                        xb[nb][j][0] = v.x; xb[nb][j][1] = v.y; xb[nb][j][2] = v.z; xb[nb][j][3] = v.w;
                                    }
                                }
                            }
                        }
                        if (FMT == 2 || !xf16) {
                            uint32_t m2 = 0;
#pragma unroll
                            for (int j = 0; j < 8; ++j)
#pragma unroll
                                for (int i = 0; i < 4; ++i) m2 = __vmaxu2(m2, xb[nb][j][i] & 0x7FFF7FFFu);
                            m2 = __vmaxu2(m2, __shfl_xor_sync(0xFFFFFFFFu, m2, 1));
                            m2 = __vmaxu2(m2, __shfl_xor_sync(0xFFFFFFFFu, m2, 2));             // the four lanes of activation row m
                            uint32_t amax = max(m2 & 0xFFFFu, m2 >> 16);
                            const uint32_t inf = xf16 ? 0x7C00u : 0x7F80u;
                            const bool bad = amax >= inf;
                            if (bad) {                                                          // rare: the largest finite magnitude sets the scale
                                amax = 0;
#pragma unroll
                                for (int j = 0; j < 8; ++j)
#pragma unroll
                                    for (int i = 0; i < 8; ++i) {
                                        const uint32_t mag = (xb[nb][j][i >> 1] >> (16 * (i & 1))) & 0x7FFFu;
                                        if (mag < inf) amax = max(amax, mag);
                                    }
                            }
                            {                                                                   // (lanes of other rows have the row's value already)
                                const uint32_t o1 = max(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
                                amax = max(o1, __shfl_xor_sync(0xFFFFFFFFu, o1, 2));
                            }
                            // power of two that brings the slice's largest magnitude to [2^14, 2^15) - 2.0-bit: [2^10, 2^11), so that the
                            // groups' sums stay in range; fp16 activations need it only there
                            constexpr int kTop = FMT == 2 ? 10 : 14;
                            int e = 0;
                            if (xf16) {
                                if (amax != 0) e = (amax < 0x400u ? -14 : (int)(amax >> 10) - 15) - kTop;
                            } else if (amax >= 0x80u) {
                                e = max(-100, (int)(amax >> 7) - 127 - kTop);
                            }
                            const float down = __uint_as_float((uint32_t)(127 - e) << 23), upg = __uint_as_float((uint32_t)(127 + e) << 23);
                            float gsum = 0.f, half_sum = 0.f;
#pragma unroll
                            for (int j = 0; j < 8; ++j) {
#pragma unroll
                                for (int i = 0; i < 4; ++i) {
                                    const uint32_t w = xb[nb][j][i];
                                    float2 f;
                                    if (xf16) f = __half22float2(*reinterpret_cast<const __half2*>(&w));
                                    else f = make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xFFFF0000u));
                                    f.x *= down; f.y *= down;
                                    xb[nb][j][i] = pack_h2(f.x, f.y);
                                    if (FMT == 2) gsum += f.x + f.y;
                                }
                                if constexpr (FMT == 2) {
                                    if (((j + 1) * 8) % G == 0) {                            // a scale group ends here
                                        const int gi = (j * 8) / G;
                                        gsum *= 0.5f;
                                        if (gi & 1) {
                                            const float h0 = __half2float(__float2half_rn(half_sum)), h1 = __half2float(__float2half_rn(gsum));
                                            xc[nb][gi >> 1][0] = pack_h2(h0, h1);
                                            xc[nb][gi >> 1][1] = pack_h2(half_sum - h0, gsum - h1);
                                        } else {
                                            half_sum = gsum;
                                        }
                                        gsum = 0.f;
                                    }
                                }
                            }
                            up[nb][0] = __shfl_sync(0xFFFFFFFFu, upg, 8 * t);          // lane (g' = 2t, *) holds activation row 2t
                            up[nb][1] = __shfl_sync(0xFFFFFFFFu, upg, 8 * t + 4);
                        }
                    }
                }
            };

            auto finish = [&](float sum, int col, int n) {                          // bias, store; returns what was stored
                if (FMT != 0 && (__float_as_uint(sum) & 0x7F800000u) == 0x7F800000u) sum = mma_dense<FMT>(P, G, x_dtype, col, n, sum);
                if (P.bias != nullptr) sum += load_any(P.bias, x_dtype, n);
                store_any(P.y, y_dtype, (int64_t)col * (P.ldy > 0 ? P.ldy : N) + n, sum);
                return sum;
            };
            // launches from a table only have peers; every lane of the warp
            auto to_peers = [&](float sum, int col, int n, int q, bool out) {
                if (kGroup && peers.world > 1) mma_store_peers(peers, P.y, y_dtype, P.ldy > 0 ? P.ldy : N, col, n, q, out, sum);
            };
            // ---- adds up an item's partial sums (pair, chunk) in buffer b ----
            auto reduce = [&](int pair, int chunk, int b) {
                float sum = 0.f;
                if (q_col < M) {
                    const int act = min(per, slices - chunk * per) - q_sub * q_per;
                    const uint32_t src = part + (uint32_t)(b * kMmaWarps + q_sub * q_per) * slot + (q_col * Sh::kPitch + q_row) * 4;
#pragma unroll 4
                    for (int w = 0; w < q_per; ++w)
                        if (w < act) sum += __uint_as_float(lds_u32(src + w * slot));
                }
                const int n = (b0 + pair * T) * 16 + q_row;
                // the low-rank term, once per output: the lanes that share one split its ranks (one lane alone took 0.4 us a rank)
                if (P.lora_rank > 0 && chunk == 0 && q_col < M && n < N) {
                    const int rank = P.lora_rank;
#pragma unroll 1
                    for (int r = q_sub; r < rank; r += 1 << qs)
                        sum = fmaf(__ldcg(P.lora_t + q_col * rank + r), mma_load16(P.lora_b, xf16, (int64_t)r * N + n), sum);
                }
                for (int o = 1; o < (1 << qs); o <<= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
                const bool out = q_sub == 0 && q_col < M && n < N && n < (b0 + nt) * 16;
                if (chunks > 1) {
                    float* a = acc_sums + (pair * M + q_col) * R + q_row;
                    if (out && chunk > cr) sum += *a;
                    if (out && (chunk + cs < chunks || cs > 1)) *a = sum;
                    if (chunk + cs < chunks || cs > 1) return;
                }
                if (out) sum = finish(sum, q_col, n);
                to_peers(sum, q_col, n, qs, out);
            };

            int pair = 0, chunk = cr, act = 0, last_pair = -1, last_chunk = 0;
            for (int n = 0; n < total; ++n) {
                asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
                __syncthreads();            // the item's data and the previous item's partial sums are visible, the previous stage is free
                issue(n + D, true);
                if (last_pair >= 0 && !dead) reduce(last_pair, last_chunk, buf ^ 1);
                uint32_t lut = base;                                  // opaque: sums with it are not worth registers of their own
                asm volatile("" : "+r"(lut));
                const uint32_t st = lut + plan.off_ring + stage * plan.stage_bytes;
                if (pair == 0) {
                    act = min(per, slices - chunk * per);
                    load_x(chunk, st);
                }
                if (!dead && warp < act) {
                    const uint32_t my_part = part + (uint32_t)(buf * kMmaWarps + warp) * slot + g * 4;
#pragma unroll
                    for (int tl = 0; tl < T; ++tl) {
                        if (T == 2 && tl == 1 && pair * 2 + 1 >= nt) break;
                        uint32_t ca = st + (tl * 16 + g) * pc + warp * F::kCode + t * (F::kCode / 4), cb = ca + 8 * pc;
                        uint32_t la = st + plan.scale_off + (tl * 16 + g) * ps + warp * F::kScale + t * (F::kScale / 4), lb = la + 8 * ps;
                        uint32_t wa[F::kCW], wb[F::kCW], sa[F::kSW], sb[F::kSW];
                        if constexpr (kRag) {                         // each row starts at its own offset inside 16 bytes
                            const uint32_t row = (uint32_t)((b0 + pair * T + tl) * 16 + g), k0 = (uint32_t)(chunk * per * 256);
                            const uint32_t oc = row * rc + code_bytes(k0), os = row * rs + k0 / G * 2;
                            ca += oc & 15u; cb += (oc + 8 * rc) & 15u;
                            la += os & 15u; lb += (os + 8 * rs) & 15u;
                            lds_words<F::kCW, FMT == 0 ? 2 : 4>(ca, wa);
                            lds_words<F::kCW, FMT == 0 ? 2 : 4>(cb, wb);
                            lds_words<F::kSW, G == 32 ? 2 : 4>(la, sa);
                            lds_words<F::kSW, G == 32 ? 2 : 4>(lb, sb);
                            const int left = K - ((chunk * per + warp) * 256 + t * 64);      // k of this lane's window inside the matrix
                            if (left < 64) {                          // scales beyond the row: 0 (x is 0 there, the scale must be finite)
#pragma unroll
                                for (int i = 0; i < F::kSW; ++i)
#pragma unroll
                                    for (int h = 0; h < 2; ++h)
                                        if ((2 * i + h) * G >= left) { sa[i] &= h ? 0x0000FFFFu : 0xFFFF0000u; sb[i] &= h ? 0x0000FFFFu : 0xFFFF0000u; }
                            }
                        } else {
                            lds_words<F::kCW, FMT == 0 ? 4 : 16>(ca, wa);
                            lds_words<F::kCW, FMT == 0 ? 4 : 16>(cb, wb);
                            lds_words<F::kSW, 16>(la, sa);
                            lds_words<F::kSW, 16>(lb, sb);
                        }
                        const uint32_t dst = my_part + tl * 64;
                        if constexpr (kI8) {
                            // chunks 0-3 of the lane belong to scale group 2t, 4-7 to group 2t + 1: four steps of two MMAs (digit pairs)
                            float og = 0.f, og8 = 0.f;                // rows g and g + 8
                            auto half_group = [&](auto htag) {
                                constexpr int H = decltype(htag)::value;
                                int c0[4], c1[4];
                                auto step = [&](auto jtag) {
                                    constexpr int J = decltype(jtag)::value;
                                    uint32_t ua, va, ub, vb;
                                    mma_digits(rank_at_8<J>(wa), lane_f, lane_v, ua, va);
                                    mma_digits(rank_at_8<J>(wb), lane_f, lane_v, ub, vb);
                                    const uint32_t a0 = lut_u32<kMmaDigitBias>(ua + lut), a2 = lut_u32<0>(va);
                                    const uint32_t a1 = lut_u32<kMmaDigitBias>(ub + lut), a3 = lut_u32<0>(vb);
                                    if constexpr ((J & 3) == 0) {
                                        mma_s8_zero(c0, a0, a1, a2, a3, xb[0][J][0], xb[0][J][1]);
                                        mma_s8_zero(c1, a0, a1, a2, a3, xb[0][J][2], xb[0][J][3]);
                                    } else {
                                        mma_s8(c0, a0, a1, a2, a3, xb[0][J][0], xb[0][J][1]);
                                        mma_s8(c1, a0, a1, a2, a3, xb[0][J][2], xb[0][J][3]);
                                    }
                                };
                                step(std::integral_constant<int, 4 * H + 0>{});
                                step(std::integral_constant<int, 4 * H + 1>{});
                                step(std::integral_constant<int, 4 * H + 2>{});
                                step(std::integral_constant<int, 4 * H + 3>{});
                                // column 2t holds digits 0 (c0) and 1 (c1), column 2t + 1 digits 2 and 3; rows g (0, 1) and g + 8 (2, 3)
                                const float sg = fmaf((float)(c0[0] * 128 + c1[0]), 16384.f, (float)(c0[1] * 128 + c1[1]));
                                const float sg8 = fmaf((float)(c0[2] * 128 + c1[2]), 16384.f, (float)(c0[3] * 128 + c1[3]));
                                const float fa = __half2float(__ushort_as_half((uint16_t)(H ? (sa[0] >> 16) : (sa[0] & 0xFFFFu))));
                                const float fb = __half2float(__ushort_as_half((uint16_t)(H ? (sb[0] >> 16) : (sb[0] & 0xFFFFu))));
                                og = fmaf(sg * up[0][H], fa * upb[H], og);
                                og8 = fmaf(sg8 * up[0][H], fb * upb[H], og8);
                            };
                            half_group(std::integral_constant<int, 0>{});
                            half_group(std::integral_constant<int, 1>{});
                            og += __shfl_xor_sync(0xFFFFFFFFu, og, 1);
                            og8 += __shfl_xor_sync(0xFFFFFFFFu, og8, 1);
                            og += __shfl_xor_sync(0xFFFFFFFFu, og, 2);
                            og8 += __shfl_xor_sync(0xFFFFFFFFu, og8, 2);
                            if (t == 0) { sts_f32(dst, og); sts_f32(dst + 32, og8); }
                        } else {
                            float acc[NB][4];
                            auto chunk8 = [&](auto jtag) {
                                constexpr int J = decltype(jtag)::value, si = J * 8 / G;
                                constexpr uint32_t sel = (si & 1) ? 0x3232u : 0x1010u;
                                uint32_t ra[4], rb[4];
                                mma_decode<FMT, J>(ra, wa, prmt(sa[si >> 1], 0u, sel), lut, lane_at, lane_f, lane_v);
                                mma_decode<FMT, J>(rb, wb, prmt(sb[si >> 1], 0u, sel), lut, lane_at, lane_f, lane_v);
#pragma unroll
                                for (int nb = 0; nb < NB; ++nb) {
                                    if constexpr (J == 0) mma_f16_zero(acc[nb], ra[0], rb[0], ra[1], rb[1], xb[nb][J][0], xb[nb][J][1]);
                                    else mma_f16(acc[nb], ra[0], rb[0], ra[1], rb[1], xb[nb][J][0], xb[nb][J][1]);
                                    mma_f16(acc[nb], ra[2], rb[2], ra[3], rb[3], xb[nb][J][2], xb[nb][J][3]);
                                }
                            };
                            chunk8(std::integral_constant<int, 0>{}); chunk8(std::integral_constant<int, 1>{});
                            chunk8(std::integral_constant<int, 2>{}); chunk8(std::integral_constant<int, 3>{});
                            chunk8(std::integral_constant<int, 4>{}); chunk8(std::integral_constant<int, 5>{});
                            chunk8(std::integral_constant<int, 6>{}); chunk8(std::integral_constant<int, 7>{});
                            if constexpr (FMT == 2) {
#pragma unroll
                                for (int i = 0; i < F::kSW; ++i)
#pragma unroll
                                    for (int nb = 0; nb < NB; ++nb) mma_f16(acc[nb], sa[i], sb[i], sa[i], sb[i], xc[nb][i][0], xc[nb][i][1]);
                            }
#pragma unroll
                            for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                                for (int c = 0; c < 2; ++c)
                                    if (col_on[nb][c]) {
                                        sts_f32(dst + (nb * 8 + 2 * t + c) * (Sh::kPitch * 4), acc[nb][c] * up[nb][c]);
                                        sts_f32(dst + (nb * 8 + 2 * t + c) * (Sh::kPitch * 4) + 32, acc[nb][2 + c] * up[nb][c]);
                                    }
                        }
                    }
                    if constexpr (kI8) {
                        if (xbad) mma_add_non_finite(x, chunk * per + warp, smem + (st - base) + lane * pc + warp * F::kCode,
                                                     reinterpret_cast<const uint16_t*>(smem + (st - base) + plan.scale_off + lane * ps + warp * F::kScale),
                                                     reinterpret_cast<float*>(smem + (part - base) + (uint32_t)(buf * kMmaWarps + warp) * slot) + lane);
                    }
                }
                last_pair = pair; last_chunk = chunk;
                if (++stage == S) stage = 0;
                if (++pair == np) { pair = 0; chunk += cs; }
                buf ^= 1;
            }
            __syncthreads();
            if (!dead && last_pair >= 0) reduce(last_pair, last_chunk, buf ^ 1);
            first_run = false;
            if (chunks == 1) break;                                   // all tiles were one block, the cluster's first CTA had its chunk and stored
            if (cs > 1) {
                // every CTA of the cluster holds its chunks' sums: each adds up a share of the outputs, chunks in CTA order
                mma_cluster_sync();
                const int ranks = min(cs, chunks);
                if (!dead)
                    for (int i = tid + cr * kMmaThreads; i - lane < np * M * R; i += cs * kMmaThreads) {
                        const int row = i % R, pm = i / R, pr = pm / M, col = pm - pr * M, n = (b0 + pr * T) * 16 + row;
                        const bool out = i < np * M * R && n < N && n < (b0 + nt) * 16;
                        float sum = 0.f;
                        if (out) {
                            for (int r = 0; r < ranks; ++r) sum += mma_ld_cluster(base + plan.off_acc + i * 4, r);
                            sum = finish(sum, col, n);
                        }
                        to_peers(sum, col, n, 0, out);
                    }
                mma_cluster_sync();         // nobody leaves, or writes these sums again, before all have read them
            }
        }
    }

    asm volatile("cp.async.wait_all;" ::: "memory");               // nothing of this thread is still in flight into shared memory
    if (tid == 0 && ctl->abort_flag != 0) {
        atomicCAS(&g_device_status, 0, ctl->abort_flag);
        if (peers.host_status != nullptr) *reinterpret_cast<volatile int*>(peers.host_status) = ctl->abort_flag;
    }
    if (signal) {
        // CTAs without work have not waited for the launch ahead: they must not arrive at a counter that it still uses
        if (overlap == 1) asm volatile("griddepcontrol.wait;" ::: "memory");
        __syncthreads();
        if (tid == 0) peer_signal(peers);
    }
    leave_after_predecessor(overlap);
}

// ---- host side ---------------------------------------------------------------------------------------------------
inline bool gemv_mma_ok(int fmt, int64_t M, int64_t N, int64_t K, int group, int x_dtype) {
    return M >= 1 && M <= 16 && N >= 1 && K >= 32 && K % 32 == 0 && K < (1 << 26) && N < (1 << 28) && N * K < (int64_t)1 << 33 &&
           (x_dtype == OJX_BF16 || x_dtype == OJX_F16) && (group == 32 || group == 16 || (group == 8 && fmt != 0));
}

// `max_per`: slices per chunk of the launch's largest item.
template <int FMT, int G, int NB, bool kRag>
inline MmaPlan mma_plan(int M, int max_per, bool chunked, int cluster) {
    using F = MmaFmt<FMT, G>;
    using Sh = MmaShape<FMT, G, NB, kRag>;
    MmaPlan p;
    p.cluster = cluster;
    auto up = [](int v) { return (v + 127) / 128 * 128; };
    p.scale_off = up(Sh::kRows * mma_pitch(max_per, F::kCode, kRag));
    p.x_off = up(p.scale_off + Sh::kRows * mma_pitch(max_per, F::kScale, kRag));
    const int x_bytes = kMmaWarps * M * 512, part = 2 * kMmaWarps * M * Sh::kPitch * 4, acc = chunked || cluster > 1 ? kMmaAccTiles * 16 * M * 4 : 0;
    for (p.x_staged = M <= kMmaXStageRows ? 1 : 0;; p.x_staged = 0) {      // x travels inside the stages where there is room
        p.stage_bytes = p.x_off + (p.x_staged ? x_bytes : 0);
        p.off_ring = up(F::kLut);
        p.off_part = p.off_ring + Sh::kStages * p.stage_bytes;
        p.off_acc = p.off_part + up(part);
        p.off_x = p.off_acc + up(acc);
        p.off_ctl = p.off_x + kMmaWarps * kMmaXBytes;
        p.total = p.off_ctl + up((int)sizeof(MmaCtl));
        if (p.total <= 227 * 1024 || !p.x_staged) break;
    }
    return p;
}

// Clusters of `size` CTAs of a kernel that fit the device at once (cached per device by the caller).
template <typename... Params>
static int mma_max_clusters(void (*kernel)(Params...), int size, size_t smem) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(num_sms() / size * size));
    cfg.blockDim = dim3(kMmaThreads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)size;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) { (void)cudaGetLastError(); n = 0; }
    return n;
}

// `units`: CTAs (clusters, when `cluster` > 1) the work can occupy.
template <int FMT, int G, int NB, bool kRag, bool kGroup, bool kI8 = false>
static int32_t mma_launch(const ojx_e8t_gemv_problem* probs, const ojx_e8t_gemv_problem& single, int units, int cluster, int max_per,
                          bool chunked, int M, int x_dtype, int y_dtype, const PeerMap& peers, int overlap, cudaStream_t s) {
    auto kernel = gemv_mma_kernel<FMT, G, NB, kRag, kGroup, kI8>;
    static std::atomic<uint64_t> configured{0};
    const int32_t st = ensure_dynamic_smem(kernel, 227 * 1024, configured);
    OJX_RETURN_IF(st != OJX_OK, st);
    int room = num_sms();
    if (cluster > 1) {
        static std::atomic<int> fit[2][64];                                    // clusters of two and of four that fit, plus one, per device
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return OJX_ERR_LAUNCH;
        std::atomic<int>& f = fit[cluster == 4][dev];
        if (f.load(std::memory_order_relaxed) == 0) f.store(mma_max_clusters(kernel, cluster, 227 * 1024) + 1, std::memory_order_relaxed);
        room = f.load(std::memory_order_relaxed) - 1;
        if (room <= 0) { cluster = 1; room = num_sms(); }
    }
    const MmaPlan plan = mma_plan<FMT, G, NB, kRag>(M, max_per, chunked, cluster);
    const int grid = (units < room ? units : room) * cluster;
    // a launch that waits for its peers reads x after them whatever it may read before the launch ahead has ended
    const bool late_x = peers.sync != nullptr && (peers.mode & OJX_GEMV_WAIT_PEERS) != 0;
    return launch_maybe_overlapped(kernel, grid, kMmaThreads, plan.total, s, overlap != 0, cluster,
                                   probs, single, M, x_dtype, y_dtype, overlap == 0 && late_x ? 1 : overlap, plan, peers);
}

// K of several chunks over few tiles: the CTAs of a cluster split the chunks, so that each prepares x for its own chunks only
// and has more tiles to spread that over.  Beyond four tiles per CTA the preparation no longer shows.
inline int mma_cluster_for(int tiles, int chunks) {
    if (chunks < 2 || tiles >= 4 * num_sms()) return 1;
    return chunks >= 4 ? 4 : 2;
}

template <int FMT, int G>
static int32_t mma_dispatch(bool rag, const ojx_e8t_gemv_problem& p, int tiles, int M, int x_dtype, int y_dtype, const PeerMap& peers, int overlap, cudaStream_t s) {
    const int per = mma_per_chunk(p.K), chunks = mma_chunks(p.K), cluster = mma_cluster_for(tiles, chunks);
    const bool chunked = chunks > 1;
    if (rag) return M <= 8 ? mma_launch<FMT, G, 1, true, false>(nullptr, p, tiles, cluster, per, chunked, M, x_dtype, y_dtype, peers, overlap, s)
                           : mma_launch<FMT, G, 2, true, false>(nullptr, p, tiles, cluster, per, chunked, M, x_dtype, y_dtype, peers, overlap, s);
    if (FMT == 0 && G == 32 && M == 1 && x_dtype == OJX_BF16)
        return mma_launch<0, 32, 1, false, false, true>(nullptr, p, tiles, cluster, per, chunked, M, x_dtype, y_dtype, peers, overlap, s);
    return M <= 8 ? mma_launch<FMT, G, 1, false, false>(nullptr, p, tiles, cluster, per, chunked, M, x_dtype, y_dtype, peers, overlap, s)
                  : mma_launch<FMT, G, 2, false, false>(nullptr, p, tiles, cluster, per, chunked, M, x_dtype, y_dtype, peers, overlap, s);
}

// One matrix; the caller has checked gemv_mma_ok and the alignment (16 bytes) of x, codes and scales.  `overlap` 3: nothing is read
// before the launch ahead has ended; 1: codes and scales may be (the launch ahead does not write them).
static int32_t gemv_mma_single(int fmt, const ojx_e8t_gemv_problem& p, int group, int64_t M, int x_dtype, int y_dtype, int overlap, cudaStream_t s) {
    PeerMap peers = peer_map_self();
    peers.host_status = host_status_device_ptr(s);
    if (wait_limit_override() != 0) peers.wait_limit = wait_limit_override();
    const bool rag = p.K % 256 != 0;
    const int tiles = (p.N + 15) / 16, m = (int)M;
#define OJX_MMA(F, GG) return mma_dispatch<F, GG>(rag, p, tiles, m, x_dtype, y_dtype, peers, overlap, s)
    if (fmt == 0 && group == 32) OJX_MMA(0, 32);
    if (fmt == 0 && group == 16) OJX_MMA(0, 16);
    if (fmt == 2 && group == 32) OJX_MMA(2, 32);
    if (fmt == 2 && group == 16) OJX_MMA(2, 16);
    if (fmt == 2 && group == 8) OJX_MMA(2, 8);
    if (fmt == 1 && group == 32) OJX_MMA(1, 32);
    if (fmt == 1 && group == 16) OJX_MMA(1, 16);
    if (fmt == 1 && group == 8) OJX_MMA(1, 8);
#undef OJX_MMA
    return OJX_ERR_UNSUPPORTED;
}

}  // namespace ojx
