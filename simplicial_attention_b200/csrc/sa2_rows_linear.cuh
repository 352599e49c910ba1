// y = x W^T for the few rows of a generation step: x [rows][k], W [outs][k] (a Linear's weight), bf16, fp32 sums.
//
// Bound: reading W once (1.6 MB for 1536 x 512, 0.25 us of HBM) - in practice the latency of a launch.  A CTA owns 16
// outputs, its eight warps take alternate 32-wide pieces of k, and the sums of the warps are added in order through
// shared memory, so a row's result does not depend on the rows beside it.  W is the 16-row operand of mma.m16n8k16 and
// eight rows of x the other one.  The order of k inside a piece is free as long as both operands share it: a thread takes
// eight consecutive values of a row, one 16-byte load, where the instruction's own order would need 4-byte loads.
// The library call cost the host 12 us (choosing a kernel per call) against 4 us for this launch, and a generation
// step of few rows is bound by the host: 59 -> 40 us with one sequence.  On the device, against the library: 512 -> 1536
// 2.1 against 3.2 us at 1 row, 2.35 against 3.0 at 16, 3.7 against 3.0 at 32; 2048 -> 6144 4.4 against 5.6, 6.5 against
// 5.6, 10.6 against 5.7.  So 16 rows are the most that sa2_rows_linear takes: there the host's 8 us outweigh the last microsecond.
// sa2_norm_linear takes up to 64, for small W (the caller's rule), and an RMSNorm of x on the way in: every CTA forms the row scales
// of all rows again (32 rows of 512: 4.7 us against 2.0 for the norm's own launch and 3.0 for the library's product, and one call on the
// host instead of two).
#pragma once
#include "sa2_headnorm.cuh"
#include <cuda_bf16.h>

namespace sa2 {
namespace rows_linear {

constexpr int WARPS = 8, OUTS = 16, MAX_ROWS = 16, MAX_NORM_ROWS = 64;

__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// RMSNorm of the rows of x on their way in, with the arithmetic and the rounding of the norm's own kernel
struct Norm { const void *gain; int bf16; float eps; };

// MT: groups of eight rows of x
template <int MT, bool NORM>
__global__ void __launch_bounds__(WARPS * 32) kernel(const __nv_bfloat16 *x, const __nv_bfloat16 *w, __nv_bfloat16 *y, int rows, int k, int outs, const Norm norm) {
    __shared__ float part[WARPS][OUTS][8 * MT + 1];
    __shared__ float rstd[NORM ? 8 * MT : 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int o0 = blockIdx.x * OUTS;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    float c[MT][4];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
        for (int z = 0; z < 4; ++z) c[m][z] = 0.f;
    const __nv_bfloat16 *w0 = w + (int64_t)(o0 + g) * k + t * 8, *w1 = w0 + (int64_t)8 * k;
    if constexpr (NORM) {
        float ss[MT];                 // of rows warp, warp + 8, ...
#pragma unroll
        for (int m = 0; m < MT; ++m) ss[m] = 0.f;
        for (int c = lane * 8; c < k; c += 256) {
            uint4 u[MT];
#pragma unroll
            for (int m = 0; m < MT; ++m) u[m] = warp + WARPS * m < rows ? __ldg(reinterpret_cast<const uint4 *>(x + (int64_t)(warp + WARPS * m) * k + c)) : zero;
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                const uint32_t p[4] = {u[m].x, u[m].y, u[m].z, u[m].w};
#pragma unroll
                for (int z = 0; z < 4; ++z) {
                    const float a = __uint_as_float(p[z] << 16), b = __uint_as_float(p[z] & 0xffff0000u);
                    ss[m] = fmaf(b, b, fmaf(a, a, ss[m]));
                }
            }
        }
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            ss[m] = headnorm::head_sum<256>(ss[m]);
            if (lane == 0) rstd[warp + WARPS * m] = rsqrtf(ss[m] / (float)k + norm.eps);
        }
        __syncthreads();
    }
    // eight values of row r of x, normalised
    auto scaled = [&](uint4 u, int r, const float (&gn)[8]) {
        const float rs = rstd[r];
        uint32_t *p = reinterpret_cast<uint32_t *>(&u);
#pragma unroll
        for (int z = 0; z < 4; ++z) {
            const __nv_bfloat162 t2 = __floats2bfloat162_rn(__uint_as_float(p[z] << 16) * rs * gn[2 * z], __uint_as_float(p[z] & 0xffff0000u) * rs * gn[2 * z + 1]);
            p[z] = *reinterpret_cast<const uint32_t *>(&t2);
        }
        return u;
    };
    // two pieces at a time, all their loads first
    for (int k0 = warp * 32; k0 < k; k0 += 2 * WARPS * 32) {
        uint4 a[2], b[2], v[2][MT];
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int kq = k0 + q * WARPS * 32;
            const bool on = kq < k;
            a[q] = on ? __ldg(reinterpret_cast<const uint4 *>(w0 + kq)) : zero;
            b[q] = on ? __ldg(reinterpret_cast<const uint4 *>(w1 + kq)) : zero;
#pragma unroll
            for (int m = 0; m < MT; ++m)
                v[q][m] = on && m * 8 + g < rows ? __ldg(reinterpret_cast<const uint4 *>(x + (int64_t)(m * 8 + g) * k + kq + t * 8)) : zero;
        }
        if constexpr (NORM) {
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const int kq = k0 + q * WARPS * 32;
                if (kq >= k) break;
                float gn[8];
                if (norm.bf16) headnorm::load8<__nv_bfloat16>(reinterpret_cast<const __nv_bfloat16 *>(norm.gain) + kq + t * 8, gn);
                else headnorm::load8<float>(reinterpret_cast<const float *>(norm.gain) + kq + t * 8, gn);
#pragma unroll
                for (int m = 0; m < MT; ++m) if (m * 8 + g < rows) v[q][m] = scaled(v[q][m], m * 8 + g, gn);
            }
        }
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                mma_bf16(c[m], a[q].x, b[q].x, a[q].y, b[q].y, v[q][m].x, v[q][m].y);
                mma_bf16(c[m], a[q].z, b[q].z, a[q].w, b[q].w, v[q][m].z, v[q][m].w);
            }
    }
#pragma unroll
    for (int m = 0; m < MT; ++m) {
        part[warp][g][m * 8 + 2 * t] = c[m][0];
        part[warp][g][m * 8 + 2 * t + 1] = c[m][1];
        part[warp][g + 8][m * 8 + 2 * t] = c[m][2];
        part[warp][g + 8][m * 8 + 2 * t + 1] = c[m][3];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < OUTS * rows; e += WARPS * 32) {
        const int r = e / OUTS, o = e % OUTS;
        float s = 0.f;
#pragma unroll
        for (int p = 0; p < WARPS; ++p) s += part[p][o][r];
        y[(int64_t)r * outs + o0 + o] = __float2bfloat16_rn(s);
    }
}

}  // namespace rows_linear
}  // namespace sa2
