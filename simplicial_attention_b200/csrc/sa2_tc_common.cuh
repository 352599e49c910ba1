// What the tcgen05 kernels share: tile sizes, fast math and packing helpers, the warp-wide bounded wait.
#pragma once
#include "sa2_common.cuh"
#include "sa2_sm100.cuh"
#include <cuda.h>
#include <math_constants.h>

namespace sa2 {
namespace tc {

using namespace sa2::sm100;

constexpr int TQ = 128;          // rows of a tile of query-side operands (TMEM lanes)
constexpr int TJ = 128;          // first-key rows per tile
constexpr uint32_t TILE_BYTES = TJ * 64 * 2;

// error bits reported through the device status word
enum { ERR_FWD_PRODUCER = 1, ERR_FWD_MMA = 2, ERR_FWD_SOFTMAX = 4, ERR_FWD_OUTPUT = 8 };

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float lg2(float x) {
    float y;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&v);
}
// a * b - hi, hi = bf16(a * b): the product of two bf16 values has 16 bits, so the pair (hi, this) is exact
__device__ __forceinline__ uint32_t mul_rest_bf16x2(uint32_t a, uint32_t b, uint32_t hi) {
    __nv_bfloat162 r = __hfma2(*reinterpret_cast<__nv_bfloat162 *>(&a), *reinterpret_cast<__nv_bfloat162 *>(&b),
                               __hneg2(*reinterpret_cast<__nv_bfloat162 *>(&hi)));
    return *reinterpret_cast<uint32_t *>(&r);
}
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {
    __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162 *>(&a), *reinterpret_cast<__nv_bfloat162 *>(&b));
    return *reinterpret_cast<uint32_t *>(&r);
}

__device__ __forceinline__ uint4 mul_rest_bf16x8(const uint4 &a, const uint4 &b, const uint4 &hi) {
    return make_uint4(mul_rest_bf16x2(a.x, b.x, hi.x), mul_rest_bf16x2(a.y, b.y, hi.y), mul_rest_bf16x2(a.z, b.z, hi.z), mul_rest_bf16x2(a.w, b.w, hi.w));
}

#ifndef SA2_WARP_WAIT_SLEEP
#define SA2_WARP_WAIT_SLEEP 64
#endif
// every lane of the warp waits; the result is uniform so that the .sync.aligned
// tcgen05 instructions that follow are never reached by a partial warp
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity, volatile int *abort_flag, int prof = -1) {
    return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, SA2_WARP_WAIT_SLEEP, prof));
}

// The lowest reference a row takes: below every finite logit, above -inf, so that logits of -inf weigh 0 and not NaN.
constexpr float LOWEST_REF = -3.4e38f;

// per-row hand-over between a softmax thread and the output thread of its row:
// [group][sweep parity][128] final reference of the sweep, then [group][128] denominator and
// [group][128] the reference it is expressed against
constexpr int FWD_STATS_FLOATS = 2 * 2 * 128 + 2 * 128 + 2 * 128;

// what two packed bf16 probabilities leave of the fp32 ones, as bf16: together they carry 16 bits
__device__ __forceinline__ uint32_t pack_rest(float p0, float p1, uint32_t hi) {
    return pack_bf16(p0 - __uint_as_float(hi << 16), p1 - __uint_as_float(hi & 0xffff0000u));
}

// exp2(c * s - ref) for 32 logits of one row -> 16 packed bf16 pairs, and the pairs of what the rounding left if SPLIT;
// returns their sum.  Columns outside (lo, hi] are masked (window / causality / sequence start).
template <bool SPLIT>
__device__ __forceinline__ float fwd_probs32(const uint32_t (&s)[32], uint32_t (&pk)[16], uint32_t (&rest)[16], float c, float ref,
                                             bool full, int col0, int lo, int hi) {
    float sum0 = 0.f, sum1 = 0.f;
    auto put = [&](int x, float p0, float p1) {
        sum0 += p0; sum1 += p1;
        pk[x >> 1] = pack_bf16(p0, p1);
        if constexpr (SPLIT) rest[x >> 1] = pack_rest(p0, p1, pk[x >> 1]);
    };
    if (full) {
        const uint64_t c2 = f2_pack(c, c), nref2 = f2_pack(-ref, -ref);
#pragma unroll
        for (int x = 0; x < 32; x += 2) {
            float a0, a1;
            f2_unpack(f2_fma(f2_pack(s[x], s[x + 1]), c2, nref2), a0, a1);
            put(x, ex2(a0), ex2(a1));
        }
    } else {
        // Valid columns are the integers in (lo, hi]: 2048 (half + 1/2 - |col - mid|) is at least 1024 inside and at most
        // -1024 outside, so the minimum with it leaves the exponents of valid cells alone and makes P exactly 0 elsewhere,
        // whatever S is there (FMA pipe instead of compares and selects on the ALU pipe; all values are exact).  A valid
        // NaN, or a logit far above the reference, gives inf and trips the slow path.
        const float mid = 1024.f * (float)(lo + 1 + hi) - 2048.f * (float)col0, half = 1024.f * (float)(hi - lo);
        const uint64_t c2 = f2_pack(c, c), nref2 = f2_pack(-ref, -ref);
#pragma unroll
        for (int x = 0; x < 32; x += 2) {
            float a0, a1;
            f2_unpack(f2_fma(f2_pack(s[x], s[x + 1]), c2, nref2), a0, a1);
            put(x, ex2(fminf(a0, half - fabsf(2048.f * x - mid))), ex2(fminf(a1, half - fabsf(2048.f * (x + 1) - mid))));
        }
    }
    return sum0 + sum1;
}

}  // namespace tc
}  // namespace sa2
