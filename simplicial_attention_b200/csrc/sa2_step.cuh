// Attention of a generation step with one new token per sequence, bf16: the per-head norms of the packed projection, the hand-over
// of the window caches and the attention of the new rows, in one launch.
//
// A CTA takes one (sequence, key/value head) and a stretch of the first keys; the stretches of a head are the CTAs of a cluster.
// It normalises the head's rows of the projection, fetches its stretch of K1 / V1 and the second keys and values from the
// caches, writes what it fetched to the new caches, and attends: a row of its products is (query head of the group, offset e),
//     S = (q * k2_{-e}) K1^T     P = exp2(c S - m)     W = P V1     out += v2_{-e} * W
// sixteen rows a warp on mma.m16n8k16, the products q * k2 and P as a bf16 value and a bf16 rest each, so that only inputs and result
// are rounded to 8 bits.  Partial outputs are merged against their maxima: rows of a warp by shuffles, warps through shared memory,
// CTAs through distributed shared memory.
//
// Bound: reading and writing the caches once (b32, 4 heads of 64, windows 512/32: 35 MB, 5.5 us of HBM); for few sequences the
// latency of a launch, of one trip to the caches and of the merges.  In its place were a launch of norms and copies and the tcgen05
// forward, which has 16 of the 128 rows of a tile live at one new row, walks a window of 512 in nine units of ~900 cycles, and with one
// sequence uses eight SMs.  8 query heads, windows 512/32: 46 -> 19 us at b32 (37 with 161 registers a thread, one CTA per SM), 21
// -> 8.7 us at b1; the whole step 64 -> 35 and 45 -> 32 us.
#pragma once
#include "sa2_headnorm.cuh"
#include "sa2_rows_linear.cuh"
#include "sa2_tc_common.cuh"
#include "sa2_simt.cuh"
#include <cooperative_groups.h>

namespace sa2 {
namespace step {

constexpr int WARPS = 8, THREADS = WARPS * 32;
constexpr int MAX_W2 = 64;          // second keys in shared memory

struct Set {
    const __nv_bfloat16 *cache;     // [b][keep][hk][d]
    int64_t sb, sn, sh;
    __nv_bfloat16 *dst;             // [b][rows][hk][d]: the last `rows` of the cached rows and the new one
    int keep, rows;
};
struct Params {
    headnorm::Gains gains;
    const __nv_bfloat16 *proj;      // [b][stride]
    int64_t stride;
    float eps, c;                   // scale * log2(e)
    Set set[4];                     // k1, k2, v1, v2
    __nv_bfloat16 *out;             // [b][hq][d]
    int hq, hk, g, w1, w2;
    int splits, chunk;              // CTAs of a head, first keys of each
};

// first keys in shared memory at a time, and CTAs of an SM (registers)
template <int D> constexpr int PIECE = D == 64 ? 256 : 128;
template <int D> constexpr int PER_SM = D == 64 ? 2 : 1;

// rows of D bf16 in shared memory, 16-byte chunks XOR-ed with the row
template <int D> __device__ __forceinline__ int sw(int row, int chunk) { return row * D + ((chunk ^ (row & 7)) << 3); }

template <int D> struct Smem {
    // pieces of K1, V1; second keys and values; the new rows (q of the group, then k1, k2, v1, v2)
    static size_t bytes(int g, int items) {
        return (size_t)2 * PIECE<D> * D * 2 + 2 * MAX_W2 * D * 2 + (g + 4) * D * 2 + (size_t)(items + g) * (D + 2) * 4;
    }
};

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(sm100::smem_u32(p)));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(sm100::smem_u32(p)));
}
__device__ __forceinline__ void fetch16(__nv_bfloat16 *dst, const __nv_bfloat16 *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sm100::smem_u32(dst)), "l"(src) : "memory");
}

// (query heads of the group) x (blocks of sixteen offsets), and how many warps share the keys of a block
struct Items { int per_head, blocks, parts; };
__host__ __device__ __forceinline__ Items items(int g, int w2) {
    Items t;
    t.per_head = (w2 + 15) / 16;
    t.blocks = g * t.per_head;
    t.parts = t.blocks >= WARPS ? 1 : t.blocks > 2 ? WARPS / t.blocks : 4;
    return t;
}

// Second values that are infinite or 2^64 and more: a W of some of the keys times one of them can be infinite of either sign where the W of
// all keys has one.  So the first CTA of a head, alone, forms W over all keys before it multiplies, against the maximum m and denominator l
// that the cluster found: a warp per offset, a product at a time (0.2 ms at windows 512/32).
template <int D>
__device__ __noinline__ void whole_rows(const Params &P, const __nv_bfloat16 *sNew, const __nv_bfloat16 *sK2, const __nv_bfloat16 *sV2, float *scratch,
                                        int head, float m, float l) {
    constexpr int CH = D / 32;                           // channels of a lane
    const Set &S1 = P.set[0], &T1 = P.set[2];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, hk = blockIdx.y, b = blockIdx.z;
    const int n1 = min(P.w1, S1.keep + 1), n2 = min(P.w2, P.set[1].keep + 1);
    auto at = [&](const __nv_bfloat16 *s, int row, int c) { return __bfloat162float(s[sw<D>(row, c >> 3) + (c & 7)]); };
    float acc[CH];
#pragma unroll
    for (int z = 0; z < CH; ++z) acc[z] = 0.f;
    for (int r = warp; r < n2; r += WARPS) {
        float a[CH], w[CH];
#pragma unroll
        for (int z = 0; z < CH; ++z) {
            const int c = lane * CH + z;
            a[z] = __bfloat162float(sNew[head * D + c]) * at(sK2, r, c);
            w[z] = 0.f;
        }
        for (int j = S1.keep + 1 - n1; j <= S1.keep; ++j) {
            const bool fresh = j == S1.keep;
            const __nv_bfloat16 *k = fresh ? sNew + P.g * D : S1.cache + b * S1.sb + (int64_t)j * S1.sn + hk * S1.sh;
            const __nv_bfloat16 *v = fresh ? sNew + (P.g + 2) * D : T1.cache + b * T1.sb + (int64_t)j * T1.sn + hk * T1.sh;
            float s = 0.f;
#pragma unroll
            for (int z = 0; z < CH; ++z) s = fmaf(a[z], __bfloat162float(k[lane * CH + z]), s);
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            const float p = tc::ex2(s * P.c - m);
#pragma unroll
            for (int z = 0; z < CH; ++z) w[z] = fmaf(p, __bfloat162float(v[lane * CH + z]), w[z]);
        }
#pragma unroll
        for (int z = 0; z < CH; ++z) acc[z] = fmaf(w[z] / l, at(sV2, r, lane * CH + z), acc[z]);
    }
#pragma unroll
    for (int z = 0; z < CH; ++z) scratch[warp * D + lane * CH + z] = acc[z];
    __syncthreads();
    for (int c = threadIdx.x; c < D; c += THREADS) {
        float o = 0.f;
        for (int w = 0; w < WARPS; ++w) o += scratch[w * D + c];
        P.out[((int64_t)b * P.hq + hk * P.g + head) * D + c] = __float2bfloat16_rn(o);
    }
    __syncthreads();
}

template <int D>
__global__ void __launch_bounds__(THREADS, PER_SM<D>) kernel(const __grid_constant__ Params P) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(128) uint8_t smem[];
    constexpr int CPR = D / 8;                           // 16-byte chunks of a row
    __nv_bfloat16 *sK = reinterpret_cast<__nv_bfloat16 *>(smem), *sV = sK + PIECE<D> * D, *sK2 = sV + PIECE<D> * D, *sV2 = sK2 + MAX_W2 * D;
    __nv_bfloat16 *sNew = sV2 + MAX_W2 * D;              // q rows of the group, then k1, k2, v1, v2
    float *part = reinterpret_cast<float *>(sNew + (P.g + 4) * D);       // [items][D + 2]: output, maximum, denominator
    const Items it = items(P.g, P.w2);
    float *own = part + it.blocks * it.parts * (D + 2);                  // [g][D + 2]

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gq = lane >> 2, t4 = lane & 3;
    const int split = blockIdx.x, hk = blockIdx.y, b = blockIdx.z;
    const Set &S1 = P.set[0], &S2 = P.set[1], &T1 = P.set[2], &T2 = P.set[3];
    const int n1 = min(P.w1, S1.keep + 1), n2 = min(P.w2, S2.keep + 1);
    const int j_begin = S1.keep + 1 - n1 + split * P.chunk, j_end = min(S1.keep + 1, j_begin + P.chunk);

    // Rows [first, first + count) of a set into shared memory; the new row and what is past the end come later.
    auto fetch = [&](const Set &s, __nv_bfloat16 *dst, int first, int count) {
        for (int x = threadIdx.x; x < count * CPR; x += THREADS) {
            const int r = x / CPR, c = x % CPR;
            if (first + r < s.keep) fetch16(dst + sw<D>(r, c), s.cache + b * s.sb + (int64_t)(first + r) * s.sn + hk * s.sh + c * 8);
        }
    };
    // Those of them that the new cache keeps, [from, to) in positions, from shared memory.
    auto keep = [&](const Set &s, const __nv_bfloat16 *src, int first, int from, int to) {
        const int drop = s.keep + 1 - s.rows;            // position of row 0 of the new cache
        for (int x = threadIdx.x; x < (to - from) * CPR; x += THREADS) {
            const int pos = from + x / CPR, c = x % CPR;
            if (pos < drop) continue;
            *reinterpret_cast<uint4 *>(s.dst + (((int64_t)b * s.rows + pos - drop) * P.hk + hk) * D + c * 8) =
                *reinterpret_cast<const uint4 *>(src + sw<D>(pos - first, c));
        }
    };

    // second keys and values: position keep - e at row n2 - 1 - e
    const int first2 = S2.keep + 1 - n2;
    fetch(S2, sK2, first2, n2);
    fetch(T2, sV2, first2, n2);
    if (j_begin < j_end) {
        fetch(S1, sK, j_begin, min(PIECE<D>, j_end - j_begin));
        fetch(T1, sV, j_begin, min(PIECE<D>, j_end - j_begin));
    }
    // the new rows, a warp each
    for (int x = warp; x < P.g + 4; x += WARPS) {
        const int set = x - P.g;                         // 0: k1, 1: k2, 2: v1, 3: v2
        const int head = set < 0 ? hk * P.g + x : P.hq + (set >= 2 ? 2 * P.hk : 0) + 2 * hk + (set & 1);
        const int c = lane * 8;
        float v[8], ss = 0.f;
        if (c < D) headnorm::load8<__nv_bfloat16>(P.proj + b * P.stride + head * D + c, v);
#pragma unroll
        for (int z = 0; z < 8; ++z) ss = c < D ? fmaf(v[z], v[z], ss) : 0.f;
        const float rs = rsqrtf(headnorm::head_sum<D>(ss) / (float)D + P.eps);
        if (c < D) {
            float gn[8];
            P.gains.get(head * D + c, D, gn);
#pragma unroll
            for (int z = 0; z < 8; ++z) v[z] = v[z] * rs * gn[z];
            headnorm::store8<__nv_bfloat16>(sNew + x * D + c, v);
        }
    }
    for (int x = threadIdx.x; x < it.blocks * it.parts * (D + 2); x += THREADS) part[x] = x % (D + 2) == D ? tc::LOWEST_REF : 0.f;

    bool whole = false;                                  // see whole_rows
    for (int j0 = j_begin; j0 < j_end; j0 += PIECE<D>) {
        const int count = min(PIECE<D>, j_end - j0);
        if (j0 > j_begin) {
            __syncthreads();                             // the last piece is no longer read
            fetch(S1, sK, j0, count);
            fetch(T1, sV, j0, count);
        }
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        // the new rows take their places, rows past the end are zeros
        if (threadIdx.x < CPR) {
            const int c = threadIdx.x;
            auto put = [&](__nv_bfloat16 *dst, int row, int set) {
                *reinterpret_cast<uint4 *>(dst + sw<D>(row, c)) = *reinterpret_cast<const uint4 *>(sNew + (P.g + set) * D + c * 8);
            };
            if (j0 + count == S1.keep + 1) { put(sK, count - 1, 0); put(sV, count - 1, 2); }
            if (j0 == j_begin) { put(sK2, n2 - 1, 1); put(sV2, n2 - 1, 3); }
        }
        uint32_t most = 0u;                              // of the exponents of the second values
        if (j0 == j_begin)
            for (int x = threadIdx.x; x < n2 * CPR; x += THREADS) {
                const int r = x / CPR, c = x % CPR;
                const uint4 u = *reinterpret_cast<const uint4 *>(r == n2 - 1 ? sNew + (P.g + 3) * D + c * 8 : sV2 + sw<D>(r, c));
                most = __vmaxu2(most, __vmaxu2(__vmaxu2(u.x & 0x7f807f80u, u.y & 0x7f807f80u), __vmaxu2(u.z & 0x7f807f80u, u.w & 0x7f807f80u)));
            }
        whole |= (most & 0xffffu) >= (191u << 7) || most >> 16 >= (191u << 7);
        const int padded = min(PIECE<D>, (count + 31) & ~31);
        for (int x = threadIdx.x; x < (padded - count) * CPR; x += THREADS) {
            const int o = sw<D>(count + x / CPR, x % CPR);
            *reinterpret_cast<uint4 *>(sK + o) = make_uint4(0u, 0u, 0u, 0u);
            *reinterpret_cast<uint4 *>(sV + o) = make_uint4(0u, 0u, 0u, 0u);
        }
        whole = __syncthreads_or(whole);
        keep(S1, sK, j0, j0, j0 + count);
        keep(T1, sV, j0, j0, j0 + count);
        if (split == 0 && j0 == j_begin) {
            keep(S2, sK2, first2, first2, S2.keep + 1);
            keep(T2, sV2, first2, first2, S2.keep + 1);
        }

        for (int item = warp; item < it.blocks * it.parts; item += WARPS) {
            const int block = item % it.blocks, pt = item / it.blocks;
            const int head = block / it.per_head, e0 = block % it.per_head * 16;
            const int steps = (padded / 32 + it.parts - 1) / it.parts, s0 = pt * steps, s1 = min(padded / 32, s0 + steps);
            if (s0 >= s1) continue;
            // rows e0 + gq and e0 + gq + 8 of the products q * k2, exact as a value and a rest
            uint32_t a[D / 16][4], ar[D / 16][4];
            const int e_lo = e0 + gq, e_hi = e_lo + 8;
            const bool ok_lo = e_lo < n2, ok_hi = e_hi < n2;
            const int r_lo = ok_lo ? n2 - 1 - e_lo : 0, r_hi = ok_hi ? n2 - 1 - e_hi : 0;
            const uint32_t *qw = reinterpret_cast<const uint32_t *>(sNew + head * D);
            auto word = [&](const __nv_bfloat16 *s, int r, int ch) { return *reinterpret_cast<const uint32_t *>(s + sw<D>(r, ch) + 2 * t4); };
#pragma unroll
            for (int k = 0; k < D / 16; ++k)
#pragma unroll
                for (int z = 0; z < 4; ++z) {
                    const int ch = 2 * k + (z >> 1);
                    const uint32_t q = qw[ch * 4 + t4], y = word(sK2, z & 1 ? r_hi : r_lo, ch);
                    a[k][z] = tc::mul_bf16x2(q, y);
                    ar[k][z] = tc::mul_rest_bf16x2(q, y, a[k][z]);
                }
            float w[D / 8][4], m_lo = tc::LOWEST_REF, m_hi = tc::LOWEST_REF, l_lo = 0.f, l_hi = 0.f;
#pragma unroll
            for (int n = 0; n < D / 8; ++n)
#pragma unroll
                for (int z = 0; z < 4; ++z) w[n][z] = 0.f;
            for (int st = s0; st < s1; ++st) {
                const int key0 = st * 32;
                float s[4][4];
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int z = 0; z < 4; ++z) s[n][z] = 0.f;
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int k = 0; k < D / 32; ++k) {
                        uint32_t kb[4];          // eight keys, channels [32 k, +32)
                        ldsm4(kb, sK + sw<D>(key0 + n * 8 + (lane & 7), 4 * k + (lane >> 3)));
#pragma unroll
                        for (int y = 0; y < 2; ++y) {
                            rows_linear::mma_bf16(s[n], ar[2 * k + y][0], ar[2 * k + y][1], ar[2 * k + y][2], ar[2 * k + y][3], kb[2 * y], kb[2 * y + 1]);
                            rows_linear::mma_bf16(s[n], a[2 * k + y][0], a[2 * k + y][1], a[2 * k + y][2], a[2 * k + y][3], kb[2 * y], kb[2 * y + 1]);
                        }
                    }
                float x_lo = m_lo, x_hi = m_hi;
#pragma unroll
                for (int n = 0; n < 4; ++n)
#pragma unroll
                    for (int z = 0; z < 4; ++z) {
                        const bool ok = key0 + n * 8 + 2 * t4 + (z & 1) < count && (z < 2 ? ok_lo : ok_hi);
                        s[n][z] = ok ? s[n][z] * P.c : -CUDART_INF_F;
                        if (z < 2) x_lo = fmaxf(x_lo, s[n][z]);
                        else x_hi = fmaxf(x_hi, s[n][z]);
                    }
#pragma unroll
                for (int o = 1; o <= 2; o <<= 1) {
                    x_lo = fmaxf(x_lo, __shfl_xor_sync(0xffffffffu, x_lo, o));
                    x_hi = fmaxf(x_hi, __shfl_xor_sync(0xffffffffu, x_hi, o));
                }
                const float f_lo = tc::ex2(m_lo - x_lo), f_hi = tc::ex2(m_hi - x_hi);
                m_lo = x_lo; m_hi = x_hi;
                l_lo *= f_lo; l_hi *= f_hi;
#pragma unroll
                for (int n = 0; n < D / 8; ++n) { w[n][0] *= f_lo; w[n][1] *= f_lo; w[n][2] *= f_hi; w[n][3] *= f_hi; }
                uint32_t p[4][2], pr[4][2];
#pragma unroll
                for (int n = 0; n < 4; ++n) {
#pragma unroll
                    for (int z = 0; z < 4; ++z) s[n][z] = tc::ex2(s[n][z] - (z < 2 ? m_lo : m_hi));
                    l_lo += s[n][0] + s[n][1];
                    l_hi += s[n][2] + s[n][3];
#pragma unroll
                    for (int z = 0; z < 2; ++z) {
                        p[n][z] = tc::pack_bf16(s[n][2 * z], s[n][2 * z + 1]);
                        pr[n][z] = tc::pack_rest(s[n][2 * z], s[n][2 * z + 1], p[n][z]);
                    }
                }
#pragma unroll
                for (int k = 0; k < 2; ++k)              // sixteen keys
#pragma unroll
                    for (int n = 0; n < D / 16; ++n) {   // sixteen channels
                        uint32_t vb[4];
                        ldsm4t(vb, sV + sw<D>(key0 + k * 16 + (lane & 15), 2 * n + (lane >> 4)));
#pragma unroll
                        for (int y = 0; y < 2; ++y) {
                            rows_linear::mma_bf16(w[2 * n + y], pr[2 * k][0], pr[2 * k][1], pr[2 * k + 1][0], pr[2 * k + 1][1], vb[2 * y], vb[2 * y + 1]);
                            rows_linear::mma_bf16(w[2 * n + y], p[2 * k][0], p[2 * k][1], p[2 * k + 1][0], p[2 * k + 1][1], vb[2 * y], vb[2 * y + 1]);
                        }
                    }
            }
            // the sixteen rows against one maximum, times their second values, added up
            float m = fmaxf(m_lo, m_hi);
#pragma unroll
            for (int o = 4; o <= 16; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
            float *dst = part + item * (D + 2);
            const float before = dst[D];
            m = fmaxf(m, before);
            const float f_lo = tc::ex2(m_lo - m), f_hi = tc::ex2(m_hi - m), f0 = tc::ex2(before - m);
            float l = l_lo * f_lo + l_hi * f_hi;
#pragma unroll
            for (int o = 1; o <= 16; o <<= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
            __syncwarp();
#pragma unroll
            for (int n = 0; n < D / 8; ++n) {
                const uint32_t v_lo = word(sV2, r_lo, n), v_hi = word(sV2, r_hi, n);
                float x0 = w[n][0] * f_lo * __uint_as_float(v_lo << 16) + w[n][2] * f_hi * __uint_as_float(v_hi << 16);
                float x1 = w[n][1] * f_lo * __uint_as_float(v_lo & 0xffff0000u) + w[n][3] * f_hi * __uint_as_float(v_hi & 0xffff0000u);
#pragma unroll
                for (int o = 4; o <= 16; o <<= 1) {
                    x0 += __shfl_xor_sync(0xffffffffu, x0, o);
                    x1 += __shfl_xor_sync(0xffffffffu, x1, o);
                }
                if (gq == 0) {
                    dst[n * 8 + 2 * t4] = dst[n * 8 + 2 * t4] * f0 + x0;
                    dst[n * 8 + 2 * t4 + 1] = dst[n * 8 + 2 * t4 + 1] * f0 + x1;
                }
            }
            if (lane == 0) {
                dst[D] = m;
                dst[D + 1] = dst[D + 1] * f0 + l;
            }
        }
    }
    __syncthreads();
    // the blocks and parts of a head, then the CTAs of the cluster
    for (int x = threadIdx.x; x < P.g * D; x += THREADS) {
        const int head = x / D, c = x % D;
        float m = tc::LOWEST_REF, l = 0.f, o = 0.f;
        for (int pt = 0; pt < it.parts; ++pt)
            for (int y = 0; y < it.per_head; ++y) m = fmaxf(m, part[(pt * it.blocks + head * it.per_head + y) * (D + 2) + D]);
        for (int pt = 0; pt < it.parts; ++pt)
            for (int y = 0; y < it.per_head; ++y) {
                const float *src = part + (pt * it.blocks + head * it.per_head + y) * (D + 2);
                const float f = tc::ex2(src[D] - m);
                o = fmaf(src[c], f, o);
                l = fmaf(src[D + 1], f, l);
            }
        own[head * (D + 2) + c] = o;
        if (c == 0) { own[head * (D + 2) + D] = m; own[head * (D + 2) + D + 1] = l; }
    }
    cl.sync();
    auto merged = [&](int head, int c, float &m, float &l) {
        float o = 0.f;
        m = tc::LOWEST_REF;
        l = 0.f;
        for (int r = 0; r < P.splits; ++r) m = fmaxf(m, cl.map_shared_rank(own, r)[head * (D + 2) + D]);
        for (int r = 0; r < P.splits; ++r) {
            const float *src = cl.map_shared_rank(own, r) + head * (D + 2);
            const float f = tc::ex2(src[D] - m);
            o = fmaf(src[c], f, o);
            l = fmaf(src[D + 1], f, l);
        }
        return o;
    };
    float m, l;
    if (whole) {
        for (int head = 0; split == 0 && head < P.g; ++head) {
            merged(head, 0, m, l);
            whole_rows<D>(P, sNew, sK2, sV2, reinterpret_cast<float *>(sK), head, m, l);
        }
    } else for (int x = split * THREADS + threadIdx.x; x < P.g * D; x += P.splits * THREADS) {
        const int head = x / D, c = x % D;
        const float o = merged(head, c, m, l);
        P.out[((int64_t)b * P.hq + hk * P.g + head) * D + c] = __float2bfloat16_rn(o / l);
    }
    cl.sync();               // no CTA leaves while its shared memory is read
}

// CTAs of a head: as many as run at the same time, with 32 keys at least.  0: launched, -1: not a shape this kernel takes.
template <int D> inline int launch(Params P, int b, int sms, cudaStream_t st) {
    const Items it = items(P.g, P.w2);
    const size_t smem = Smem<D>::bytes(P.g, it.blocks * it.parts);
    if (smem > 227 * 1024 / PER_SM<D> - 1024) return -1;
    const int n1 = P.w1 < P.set[0].keep + 1 ? P.w1 : P.set[0].keep + 1;
    P.splits = 1;
    while (P.splits < 8 && (int64_t)b * P.hk * P.splits * 2 <= PER_SM<D> * sms && n1 > 32 * P.splits) P.splits *= 2;
    P.chunk = (n1 + P.splits - 1) / P.splits;
    return simt::launch_clusters(kernel<D>, dim3(P.splits, P.hk, b), THREADS, smem, P.splits, st, P) ? 0 : 1;
}

}  // namespace step
}  // namespace sa2
