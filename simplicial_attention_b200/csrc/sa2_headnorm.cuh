// Per-head RMSNorm of a packed projection, forward and backward, and the hand-over of a normalised projection to
// the window caches of generation.
//
// The reference's module normalises q, k, k', v, v' per head with five separate
// RMSNorm modules after splitting the fused projection (simplicial_mha.py:124-127).
// Here the whole projection [rows][channels] is normalised in one pass: every
// group of d consecutive channels is one head.
//
//   y[r, c]  = x[r, c] * rstd[r, g] * gain(c),  rstd[r, g] = rsqrt(mean_{c in g} x^2 + eps)
//   dx       = rstd * (gy - xh * mean_g(gy * xh)),  gy = dy * gain,  xh = x * rstd
//   dgain    = sum over rows (and the heads that share it) of dy * xh
//
// The gain of a channel comes from a table with one entry per channel, or from the five gain vectors of the module
// themselves (`Gains`): no tiled copy of them is made per call, and their gradients leave the reduction summed
// over the heads.
//
// HBM-bound: every element is read once and written once, 16 bytes (eight bf16) per lane and access - a warp holds
// 256 channels, four heads of 64 at a time (with two elements per lane and access, b16 n1024 of 1536 bf16 channels
// took 54 us forward and 85 us backward; the floors are 15 and 23 us).  In the backward a lane keeps the gain
// gradient of its channels in registers over all rows of its CTA; the CTA writes one partial row and a second
// kernel adds the partial rows in a fixed order, without atomics.
#pragma once
#include "sa2_common.cuh"
#include <cuda_bf16.h>

namespace sa2 {
namespace headnorm {

constexpr int VEC = 8;                    // channels per lane and access
constexpr int WARPS = 8;                  // rows per partial row at small sizes: see headnorm_grid

template <typename T> __device__ __forceinline__ void load8(const T *p, float (&v)[8]);
template <> __device__ __forceinline__ void load8<float>(const float *p, float (&v)[8]) {
    const float4 a = *reinterpret_cast<const float4 *>(p), b = *reinterpret_cast<const float4 *>(p + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
template <> __device__ __forceinline__ void load8<__nv_bfloat16>(const __nv_bfloat16 *p, float (&v)[8]) {
    const uint4 u = *reinterpret_cast<const uint4 *>(p);
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        v[2 * z] = __uint_as_float(w[z] << 16);
        v[2 * z + 1] = __uint_as_float(w[z] & 0xffff0000u);
    }
}
template <typename T> __device__ __forceinline__ void store8(T *p, const float (&v)[8]);
template <> __device__ __forceinline__ void store8<float>(float *p, const float (&v)[8]) {
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<float4 *>(p + 4) = make_float4(v[4], v[5], v[6], v[7]);
}
template <> __device__ __forceinline__ void store8<__nv_bfloat16>(__nv_bfloat16 *p, const float (&v)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int z = 0; z < 4; ++z) {
        const __nv_bfloat162 t = __floats2bfloat162_rn(v[2 * z], v[2 * z + 1]);
        w[z] = *reinterpret_cast<const uint32_t *>(&t);
    }
    *reinterpret_cast<uint4 *>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}
// rows whose base or stride is not a multiple of 16 bytes: element by element
template <typename T> __device__ __forceinline__ void load8u(const T *p, bool aligned, float (&v)[8]) {
    if (aligned) { load8<T>(p, v); return; }
#pragma unroll
    for (int z = 0; z < 8; ++z) v[z] = (float)p[z];
}
template <typename T> __device__ __forceinline__ void store8u(T *p, bool aligned, const float (&v)[8]) {
    if (aligned) { store8<T>(p, v); return; }
#pragma unroll
    for (int z = 0; z < 8; ++z) p[z] = (T)v[z];
}

// Gain vectors.  table != null: one fp32 entry per channel.  Otherwise head h of the projection takes
//   h < hq: p[0];   hq <= h < hq + 2 hk: p[1 + ((h - hq) & 1)];   above: p[3 + ((h - hq) & 1)]
// (each key/value head's slice holds its two sets side by side), d entries each, fp32 or bf16.
struct Gains {
    const float *table;
    const void *p[5];
    int bf16, hq, hk, al;      // al: the table is 16-byte aligned (vectors always are)
    __device__ __forceinline__ int which(int h) const { return h < hq ? 0 : ((h - hq) & 1) + (h < hq + 2 * hk ? 1 : 3); }
    __device__ __forceinline__ void get(int c, int d, float (&v)[8]) const {
        if (table) {
            load8u<float>(table + c, al, v);
        } else {
            const void *src = p[which(c / d)];
            if (bf16) load8<__nv_bfloat16>(reinterpret_cast<const __nv_bfloat16 *>(src) + c % d, v);
            else load8<float>(reinterpret_cast<const float *>(src) + c % d, v);
        }
    }
};

struct Params {
    const void *x;        // [rows][x_stride], channels contiguous
    const void *dy;       // backward only: [rows][dy_stride]
    Gains gains;
    void *y;              // forward: [rows][y_stride]; backward: dx
    float *rstd;          // [rows][groups] (forward: may be null)
    float *partial;       // backward: [gridDim.x][channels]
    int64_t rows, x_stride, y_stride, dy_stride;
    int channels;
    float eps;
    int x_al, y_al, dy_al;      // rows of x / y / dy start on 16-byte boundaries
    int partial_al;             // so do those of partial (the caller's scratch has no alignment rule)
};

// sum over the lanes that share a head: D / 8 of them, all 32 for D >= 256
template <int D> __device__ __forceinline__ float head_sum(float v) {
    constexpr int LPH = D / VEC < 32 ? D / VEC : 32;
#pragma unroll
    for (int o = LPH / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// A warp covers SEG<D> = 256 CPL channels of a row; lane l holds channels 8 l + 256 k, k < CPL.
template <int D> struct Seg {
    static constexpr int CPL = D <= 256 ? 1 : D / 256;
    static constexpr int CH = 256 * CPL;
};

template <typename TX, typename TY, int D>
__global__ void __launch_bounds__(256) fwd_kernel(const Params P) {
    constexpr int CPL = Seg<D>::CPL;
    const int lane = threadIdx.x & 31;
    const int segs = (P.channels + Seg<D>::CH - 1) / Seg<D>::CH, groups = P.channels / D;
    const int64_t items = P.rows * segs;
    for (int64_t it = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); it < items; it += (int64_t)gridDim.x * 8) {
        const int64_t r = it / segs;
        const int c0 = (int)(it % segs) * Seg<D>::CH + lane * VEC;
        const bool on = c0 < P.channels;
        float v[CPL][8], ss = 0.f;
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
#pragma unroll
            for (int z = 0; z < 8; ++z) v[k][z] = 0.f;
            if (on) load8u<TX>(reinterpret_cast<const TX *>(P.x) + r * P.x_stride + c0 + 256 * k, P.x_al, v[k]);
#pragma unroll
            for (int z = 0; z < 8; ++z) ss = fmaf(v[k][z], v[k][z], ss);
        }
        const float rs = rsqrtf(head_sum<D>(ss) / (float)D + P.eps);
        if (!on) continue;
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
            float g[8];
            P.gains.get(c0 + 256 * k, D, g);
#pragma unroll
            for (int z = 0; z < 8; ++z) v[k][z] = v[k][z] * rs * g[z];
            store8u<TY>(reinterpret_cast<TY *>(P.y) + r * P.y_stride + c0 + 256 * k, P.y_al, v[k]);
        }
        if (P.rstd && (lane & (D / VEC < 32 ? D / VEC - 1 : 31)) == 0) P.rstd[r * groups + c0 / D] = rs;
    }
}

// blockDim = 32 x (warps per row) x (rows at a time); CTA x walks rows x, x + gridDim.x, ... (rows-at-a-time each)
template <typename TX, typename TY, int D>
__global__ void __launch_bounds__(Seg<D>::CPL == 1 ? 1024 : 512) bwd_kernel(const Params P) {
    constexpr int CPL = Seg<D>::CPL;
    extern __shared__ float acc[];                     // [rows at a time - 1][channels]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int segs = (P.channels + Seg<D>::CH - 1) / Seg<D>::CH, groups = P.channels / D;
    const int seg = warp % segs, rl = warp / segs, rpc = (blockDim.x >> 5) / segs;
    const int c0 = seg * Seg<D>::CH + lane * VEC;
    const bool on = c0 < P.channels;
    float g[CPL][8], dg[CPL][8];
#pragma unroll
    for (int k = 0; k < CPL; ++k) {
#pragma unroll
        for (int z = 0; z < 8; ++z) { g[k][z] = 0.f; dg[k][z] = 0.f; }
        if (on) P.gains.get(c0 + 256 * k, D, g[k]);
    }
    for (int64_t r = (int64_t)blockIdx.x * rpc + rl; r < P.rows; r += (int64_t)gridDim.x * rpc) {
        const float rs = on ? P.rstd[r * groups + c0 / D] : 0.f;
        float xh[CPL][8], gy[CPL][8], dot = 0.f;
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
            float t[8];
#pragma unroll
            for (int z = 0; z < 8; ++z) { xh[k][z] = 0.f; t[z] = 0.f; }
            if (on) {
                load8u<TX>(reinterpret_cast<const TX *>(P.x) + r * P.x_stride + c0 + 256 * k, P.x_al, xh[k]);
                load8u<TY>(reinterpret_cast<const TY *>(P.dy) + r * P.dy_stride + c0 + 256 * k, P.dy_al, t);
            }
#pragma unroll
            for (int z = 0; z < 8; ++z) {
                xh[k][z] *= rs;
                gy[k][z] = t[z] * g[k][z];
                dot = fmaf(gy[k][z], xh[k][z], dot);
                dg[k][z] = fmaf(t[z], xh[k][z], dg[k][z]);
            }
        }
        const float m = head_sum<D>(dot) / (float)D;
        if (!on) continue;
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
#pragma unroll
            for (int z = 0; z < 8; ++z) gy[k][z] = rs * (gy[k][z] - xh[k][z] * m);
            store8u<TX>(reinterpret_cast<TX *>(P.y) + r * P.y_stride + c0 + 256 * k, P.y_al, gy[k]);
        }
    }
    if (rl > 0 && on) {
#pragma unroll
        for (int k = 0; k < CPL; ++k) store8<float>(acc + (size_t)(rl - 1) * P.channels + c0 + 256 * k, dg[k]);
    }
    __syncthreads();
    if (rl == 0 && on) {
#pragma unroll
        for (int k = 0; k < CPL; ++k) {
            for (int o = 0; o < rpc - 1; ++o) {
                float t[8];
                load8<float>(acc + (size_t)o * P.channels + c0 + 256 * k, t);
#pragma unroll
                for (int z = 0; z < 8; ++z) dg[k][z] += t[z];
            }
            store8u<float>(P.partial + (size_t)blockIdx.x * P.channels + c0 + 256 * k, P.partial_al, dg[k]);
        }
    }
}

// Sum of the partial rows.  A CTA of 32 channels x 32 slices: slice j adds rows j, j + 32, ... in order, then the
// slice sums are added in order - a fixed summation tree.  With gain vectors (P.gains.table == null) CTA (x, y) adds
// channels [32 x, +32) of every head that shares vector y and stores in the vectors' type.
struct GainGrads { void *p[5]; int bf16; };
__global__ void __launch_bounds__(1024) dgain_reduce_kernel(const float *partial, float *dtable, GainGrads grads, Gains gains,
                                                            int nparts, int channels, int d) {
    __shared__ float part[32][33];
    const int lane = threadIdx.x & 31, slice = threadIdx.x >> 5;
    const int c = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (dtable) {
        if (c < channels)
            for (int p = slice; p < nparts; p += 32) s += partial[(size_t)p * channels + c];
    } else {
        const int v = blockIdx.y;
        const int h0 = v == 0 ? 0 : gains.hq + (v >= 3 ? 2 * gains.hk : 0) + ((v - 1) & 1), step = v == 0 ? 1 : 2;
        const int heads = v == 0 ? gains.hq : gains.hk;
        for (int x = slice; x < nparts * heads; x += 32) {
            const int p = x / heads, h = h0 + step * (x % heads);
            s += partial[(size_t)p * channels + h * d + c];
        }
    }
    part[slice][lane] = s;
    __syncthreads();
    if (slice == 0) {
        float t = 0.f;
#pragma unroll
        for (int j = 0; j < 32; ++j) t += part[j][lane];
        if (dtable) {
            if (c < channels) dtable[c] = t;
        } else if (grads.bf16) {
            reinterpret_cast<__nv_bfloat16 *>(grads.p[blockIdx.y])[c] = __float2bfloat16_rn(t);
        } else {
            reinterpret_cast<float *>(grads.p[blockIdx.y])[c] = t;
        }
    }
}

// ---------------------------------------------------------------------------
// Generation: normalise the projection of n new rows and put it behind the cached rows of the four key/value
// sets.  q goes to [b][n][hq][d]; set s goes to rows [keep_s, keep_s + n) of dst_s [b][keep_s + n][hk][d], whose
// first keep_s rows are copied from the cache (arbitrary batch / row / head strides, 16-byte aligned).  One launch
// in place of the norm, four concatenations and their index arithmetic on the host.
// ---------------------------------------------------------------------------
struct AppendSet {
    const void *cache;
    int64_t sb, sn, sh;     // element strides of the cache
    void *dst;
    int keep;
};
struct AppendParams {
    Params norm;            // x, gains, eps, rows = b * n; y = q
    AppendSet set[4];       // k1, k2, v1, v2
    int b, n, hq, hk;
    int norm_items;         // (row, segment) pairs, one warp each
    int64_t copy_items;     // 16-byte pieces of all four caches
};

template <typename T, int D>
__global__ void __launch_bounds__(256) append_kernel(const AppendParams A) {
    const Params &P = A.norm;
    const int lane = threadIdx.x & 31;
    const int segs = (P.channels + 255) / 256, norm_blocks = (A.norm_items + 7) / 8;
    if ((int)blockIdx.x < norm_blocks) {
        const int it = blockIdx.x * 8 + (threadIdx.x >> 5);
        if (it >= A.norm_items) return;
        const int r = it / segs, c = (it % segs) * 256 + lane * VEC;
        const bool on = c < P.channels;
        float v[8], ss = 0.f;
#pragma unroll
        for (int z = 0; z < 8; ++z) v[z] = 0.f;
        if (on) load8u<T>(reinterpret_cast<const T *>(P.x) + (int64_t)r * P.x_stride + c, P.x_al, v);
#pragma unroll
        for (int z = 0; z < 8; ++z) ss = fmaf(v[z], v[z], ss);
        const float rs = rsqrtf(head_sum<D>(ss) / (float)D + P.eps);
        if (!on) return;
        float g[8];
        P.gains.get(c, D, g);
#pragma unroll
        for (int z = 0; z < 8; ++z) v[z] = v[z] * rs * g[z];
        const int h = c / D, ch = c % D;
        if (h < A.hq) {
            store8<T>(reinterpret_cast<T *>(P.y) + ((int64_t)r * A.hq + h) * D + ch, v);
        } else {
            const int x = h - A.hq, set = (x & 1) + (x < 2 * A.hk ? 0 : 2), head = (x % (2 * A.hk)) >> 1;
            const AppendSet &S = A.set[set];
            const int bi = r / A.n, i = r % A.n;
            store8<T>(reinterpret_cast<T *>(S.dst) + (((int64_t)bi * (S.keep + A.n) + S.keep + i) * A.hk + head) * D + ch, v);
        }
        return;
    }
    constexpr int PIECES = D * (int)sizeof(T) / 16, EPP = 16 / (int)sizeof(T);       // 16-byte pieces of a head's row
    const int64_t row_pieces = (int64_t)A.hk * PIECES;
    for (int64_t x = (int64_t)(blockIdx.x - norm_blocks) * 256 + threadIdx.x; x < A.copy_items; x += (int64_t)(gridDim.x - norm_blocks) * 256) {
        int64_t y = x;
        int s = 0;
        for (; s < 3; ++s) {
            const int64_t own = (int64_t)A.b * A.set[s].keep * row_pieces;
            if (y < own) break;
            y -= own;
        }
        const AppendSet &S = A.set[s];
        const int p = (int)(y % PIECES);
        y /= PIECES;
        const int head = (int)(y % A.hk);
        y /= A.hk;
        const int row = (int)(y % S.keep), bi = (int)(y / S.keep);
        const T *src = reinterpret_cast<const T *>(S.cache) + bi * S.sb + row * S.sn + head * S.sh + p * EPP;
        T *dst = reinterpret_cast<T *>(S.dst) + (((int64_t)bi * (S.keep + A.n) + row) * A.hk + head) * D + p * EPP;
        *reinterpret_cast<uint4 *>(dst) = __ldg(reinterpret_cast<const uint4 *>(src));
    }
}

}  // namespace headnorm
}  // namespace sa2
