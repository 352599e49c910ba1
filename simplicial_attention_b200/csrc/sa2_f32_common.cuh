// fp32 tensors on the bf16 tensor cores: what the kernels of sa2_f32_fwd.cuh and sa2_f32_bwd.cuh share.
//
// Every fp32 operand x is three bf16 values, h = bf16(x), m = bf16(x - h), l = x - h - m, which carry all 24 bits of it, and a
// product of two operands is the six products of their terms that are not below 2^-24 of it: h h, h m, m h, m m, h l, l h,
// the small ones first.  The tensor cores truncate as they accumulate, so no accumulator lives longer than one unit of 64
// keys (four K steps of the large product): the sums over a window, over the offsets and over the heads are fp32 additions
// in registers.  Errors against 64 bits, norm of the difference over norm of the result, scalar fp32 kernels of sa2_simt.cuh
// against these: b1 n1000 d64 w512/32 out 2.8e-7 -> 1.3e-7, dq 5.9e-7 -> 4.1e-7, dk1 1.7e-6 -> 4.4e-7, dv1 1.5e-6 -> 3.0e-7, dk2
// 5.9e-7 -> 4.1e-7, dv2 3.7e-7 -> 2.6e-7, lse 5.0e-8 -> 5.0e-8; b1 n128 h2 d32, full causal, dk1 7.1e-7 -> 3.7e-7.
//
// Operands are made by the kernels from plain fp32 rows (any 16-byte aligned strides): no tensor maps and no scratch.
//
// Three bf16 terms are not every fp32 value: from 3.39e38 the first one is infinite (and the second a NaN, as those of infinities
// are), below 2^-109 the last ones leave bf16's range.  Where an operand's largest entry in a CTA is not in [2^-80, 2^60), or an output
// is not finite, the scalar kernels, launched behind these, do the work again: the forward's row tile by row tile (LSE_REDO), the backward's
// batch element by batch element (a flag in the workspace).  Otherwise they return at once, and since
// their blocks may take their places while the kernel before ends, a pass is 2 us longer forward and 3 both ways (4 and 6 without that; b1
// n128 h2 d32).  The maxima ride with the
// splitting of the operands, four instructions to its forty; a check of every entry for itself cost 5 to 11 % of a kernel.
#pragma once
#include "sa2_tc_common.cuh"

namespace sa2 {
namespace f32 {

using namespace sa2::sm100;
using sa2::tc::ex2;
using sa2::tc::pack_bf16;
using sa2::tc::warp_wait;

constexpr int ROWS = 128;         // rows of a tile: TMEM lanes
constexpr int UNIT = 64;          // columns of a logit tile
constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;
// error bits of the device status word
enum { ERR_FWD = 1 << 17, ERR_BWD = 1 << 18 };

// The three terms of an operand tile in shared memory, rows of 128 bytes with the 128-byte swizzle: a tile per term, or at
// head dim 32 h and m side by side and l in a second tile.
template <int D> struct Planes {
    static constexpr int TILES = D == 32 ? 2 : 3;
    __host__ __device__ static constexpr uint32_t bytes(int rows) { return (uint32_t)(TILES * rows * 128); }
    __host__ __device__ static constexpr uint32_t at(int rows, int term) {
        return D == 32 ? (uint32_t)((term >> 1) * rows * 128 + (term & 1) * 64) : (uint32_t)(term * rows * 128);
    }
};

// two values -> their three terms, packed
__device__ __forceinline__ void split2(float x0, float x1, uint32_t &h, uint32_t &m, uint32_t &l) {
    const uint64_t minus = f2_pack(-1.f, -1.f);
    h = pack_bf16(x0, x1);
    const uint64_t r = f2_fma(f2_from_bf16x2(h), minus, f2_pack(x0, x1));
    float a, b;
    f2_unpack(r, a, b);
    m = pack_bf16(a, b);
    f2_unpack(f2_fma(f2_from_bf16x2(m), minus, r), a, b);
    l = pack_bf16(a, b);
}

// the largest magnitude among `most` and eight values, NaN if there is one
__device__ __forceinline__ float most_of(float most, const float (&x)[8]) {
#pragma unroll
    for (int z = 0; z < 8; z += 2) asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(most) : "f"(x[z]), "f"(x[z + 1]));
    return most;
}
// is it one that three terms do not represent?  (0: nothing but zeros)
__device__ __forceinline__ bool out_of_range(float most) { return !(most < 1.1529215e18f) || (most > 0.f && most < 8.2718061e-25f); }
// from the threads of a warp to a word of shared memory that starts at 0 (bits of magnitudes are ordered, a NaN comes last)
__device__ __forceinline__ void put_most(uint32_t *word, float most) {
    const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(most));
    if ((threadIdx.x & 31) == 0) atomicMax(word, m);
}

// eight channels (chunk `chunk`) of row r of an operand tile of `rows` rows; `most` is the operand's largest magnitude so far
template <int D>
__device__ __forceinline__ void put8(uint8_t *tile, int rows, int r, int chunk, const float (&x)[8], float &most) {
    most = most_of(most, x);
    uint32_t h[4], m[4], l[4];
#pragma unroll
    for (int z = 0; z < 4; ++z) split2(x[2 * z], x[2 * z + 1], h[z], m[z], l[z]);
    const uint32_t o = sw128_offset(r, chunk);
    *reinterpret_cast<uint4 *>(tile + o) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4 *>(tile + (D == 32 ? sw128_offset(r, chunk + 4) : rows * 128 + o)) = make_uint4(m[0], m[1], m[2], m[3]);
    *reinterpret_cast<uint4 *>(tile + (D == 32 ? rows * 128 : 2 * rows * 128) + o) = make_uint4(l[0], l[1], l[2], l[3]);
}

__device__ __forceinline__ void load8(float (&x)[8], const float *p, bool ok) {
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (ok) {
        a = __ldg(reinterpret_cast<const float4 *>(p));
        b = __ldg(reinterpret_cast<const float4 *>(p) + 1);
    }
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
__device__ __forceinline__ const float *row_ptr(const TensorRef &t, int b, int n, int h) {
    return reinterpret_cast<const float *>(t.p) + elem_off(t, b, n, h);
}

// The six products of two operands, the smallest first: terms (l h) (h l) (m m) (m h) (h m) (h h)
__host__ __device__ constexpr int term_a(int t) { return t == 0 ? 2 : t == 2 || t == 3 ? 1 : 0; }
__host__ __device__ constexpr int term_b(int t) { return t == 1 ? 2 : t == 2 || t == 4 ? 1 : 0; }

// d[128 x 64] = A B^T over the D channels: A [128 rows], B [64 rows], both K-major in shared memory.  SWAP: the products in the order of
// B A^T, for a transposed tile of the same bits (which large logits need: their logsumexp is subtracted).
template <int D, bool SWAP = false>
__device__ __forceinline__ void issue_nt(uint32_t d, uint64_t a, uint64_t b) {
    constexpr uint32_t IDESC = idesc_bf16(128, 64, false, false);
#pragma unroll
    for (int t = 0; t < 6; ++t)
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
            mma_ss(d, a + (Planes<D>::at(ROWS, SWAP ? term_b(t) : term_a(t)) >> 4) + 2 * k,
                   b + (Planes<D>::at(UNIT, SWAP ? term_a(t) : term_b(t)) >> 4) + 2 * k, IDESC, t + k > 0);
}
// TMEM column of term `term` of the 16 keys [16 k, +16) within a region of 96 columns
__host__ __device__ constexpr uint32_t term_col(int term, int k) { return (uint32_t)(k * 24 + term * 8); }
// d[128 x D] = P B over 64 keys: P [128 x 64] in TMEM, B [64 rows] in shared memory.  Head dim 32: the products with h and m
// of B, which share its rows, land in columns [0, 32) and [32, 64), whose sum is the result.
template <int D>
__device__ __forceinline__ void issue_pv(uint32_t d, uint32_t p, uint64_t b) {
    constexpr uint32_t N64 = idesc_bf16(128, 64, false, true), N32 = idesc_bf16(128, 32, false, true);
    if constexpr (D == 32) {
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_ts(d, p + term_col(1, k), b + 128 * k, N64, k > 0);
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_ts(d, p + term_col(2, k), b + 128 * k, N32, 1u);
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_ts(d, p + term_col(0, k), b + (UNIT * 128 >> 4) + 128 * k, N32, 1u);
#pragma unroll
        for (int k = 0; k < 4; ++k) mma_ts(d, p + term_col(0, k), b + 128 * k, N64, 1u);
    } else {
#pragma unroll
        for (int t = 0; t < 6; ++t)
#pragma unroll
            for (int k = 0; k < 4; ++k)
                mma_ts(d, p + term_col(term_a(t), k), b + (Planes<D>::at(UNIT, term_b(t)) >> 4) + 128 * k, N64, t + k > 0);
    }
}
// A region of 96 columns holds a logit tile in [16, 80).  The terms of its columns [16 k, +16) go to [24 k, +24): over columns that
// have been read if those of either half are taken from the outside in, k = 0, 1 and k = 3, 2.
constexpr uint32_t LOGITS = 16;
__device__ __forceinline__ void put_terms(uint32_t region, int k, const uint32_t (&x)[16]) {
    uint32_t h[8], m[8], l[8];
#pragma unroll
    for (int z = 0; z < 8; ++z) split2(__uint_as_float(x[2 * z]), __uint_as_float(x[2 * z + 1]), h[z], m[z], l[z]);
    tmem_st8(region + 24 * k, h);
    tmem_st8(region + 24 * k + 8, m);
    tmem_st8(region + 24 * k + 16, l);
}
// the values of columns [16 k, +16), from their terms (exact)
__device__ __forceinline__ void get_terms(uint32_t region, int k, uint32_t (&x)[16]) {
    uint32_t w[16], l[16];         // (the load of l takes eight columns more than its own)
    tmem_ld16(region + 24 * k, w);
    tmem_ld16(region + 24 * k + 8, l);
    tmem_wait_ld(w);
    tmem_wait_ld(l);
#pragma unroll
    for (int z = 0; z < 8; ++z) {
        float a, b;
        f2_unpack(f2_add(f2_add(f2_from_bf16x2(l[8 + z]), f2_from_bf16x2(w[8 + z])), f2_from_bf16x2(w[z])), a, b);
        x[2 * z] = __float_as_uint(a);
        x[2 * z + 1] = __float_as_uint(b);
    }
}
// sum[] += the D columns of an accumulator (pairs of channels)
template <int D>
__device__ __forceinline__ void add_acc(uint32_t cols, uint64_t (&sum)[D / 2]) {
#pragma unroll
    for (int c = 0; c < 64; c += 32) {
        uint32_t t[32];
        tmem_ld32(cols + c, t);
        tmem_wait_ld(t);
#pragma unroll
        for (int z = 0; z < 16; ++z) {
            uint64_t &s = sum[(D == 32 ? 0 : c / 2) + z];
            s = f2_add(s, f2_pack(t[2 * z], t[2 * z + 1]));
        }
    }
}

// valid columns [lo, hi] of a logit row as the unsigned test x - lo <= len; none if hi < lo
__device__ __forceinline__ void column_range(int &lo, int hi, uint32_t &len) {
    if (hi < lo) { lo = 64; hi = 64; }
    len = (uint32_t)(hi - lo);
}

}  // namespace f32
}  // namespace sa2
