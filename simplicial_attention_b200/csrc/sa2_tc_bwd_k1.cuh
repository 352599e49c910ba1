// Backward kernel for dK1 / dV1 on tcgen05 tensor cores (bf16 operands, fp32
// accumulation in TMEM, head dims 32 and 64).
//
// One CTA owns 128 rows j of K1/V1 of one (batch, kv head); the tile stays in
// shared memory and dK1/dV1 for those rows accumulate in TMEM for the whole
// kernel, without atomics.  The CTA walks over every (query head of the group,
// query tile I, offset e) that can see its keys, or over its share of them.  Per step the builder warps form
//     A_e[i,:] = q_i * k2_{i-e}      B_e[i,:] = dO_i * v2_{i-e}      (bf16)
// and the tensor cores compute, in units of 64 query columns,
//     S^T  = K1 A_e^T       dP^T = V1 B_e^T          (rows j, columns i)
// the compute warps (one thread per key row j) turn them into
//     P^T = exp2(c S^T - lse2_i)      G^T = P^T * (dP^T - D_i)
// written back to TMEM as bf16, which then feed as A operands
//     dV1 += P^T B_e        dK1 += G^T A_e           (B_e / A_e as MN-major B)
// The same shared-memory tile is the K-major B operand of the first product
// and the MN-major B operand of the second.
//
// The per-query statistics are folded into the tensor-core products: every query row carries
// -lse2_i / c and -D_i, each split into three bf16 terms, in a small extra tile, and a constant tile
// of ones on the key side adds them with one more K=16 MMA, so that the accumulators already hold
// S^T - lse2 / c and dP^T - D and the compute threads need no per-column loads.
//
// Warps (640 threads, five aligned warpgroups with register hand-over): 0 TMA producer, then issuer of the second
// products (dV1, dK1: one issuer, which keeps the summation order fixed); 1 TMEM owner and issuer of S^T; 2 issuer of
// dP^T; 3 idle; 4-7 and 8-11 compute groups of the even and the odd units; 12-19 builders, two threads per query row.
// TMEM columns: buffer x -> S^T [128x, +64), dP^T [128x+64, +64), three buffers in flight; P^T / G^T (bf16) overwrite the
// first half of the S^T / dP^T columns they come from (at head dim 32, with their rests, all of them), so a buffer is busy until the second products of its unit are
// done; dK1 [384,448); dV1 [448,512).
//
// Bound: the exponent passes of the two groups (512 MUFU cycles per unit and scheduler) next to ~740 cycles of products
// and ~1700 cycles of shared-memory traffic per step of two units.  With a buffer per group, P^T / G^T in columns of
// their own and four builder warps a group waited 1100 of 2800 cycles a step for its next S^T: the products of a unit
// could start only when the group had finished the last (b4 n4096 h8 d64 w512/32: 1.59 -> 1.31 ms, and 1.27 with two
// columns per instruction in the exponent pass).
//
// The offsets may be split over several CTAs per key tile (consecutive ranges): a short sequence has few key tiles, and
// with grouped-query heads each walks over every head of its group.  The splits write fp32 partials, which the
// reduction of the dQ/dK2/dV2 kernel adds in order.  k1_split() picks the number.  (Splits as the CTAs of a cluster,
// added through distributed shared memory, cost 20 to 35 % at large grids: a cluster waits for its SMs to be free
// together.)  Measured: b1 n3001 h8/2 d64 w1024/16 0.78 -> 0.29 ms, b2 n128 h4 d64 w64/32 58 -> 16 us.
#pragma once
#include "sa2_tc_common.cuh"

namespace sa2 {
namespace tc {

constexpr int BK1_THREADS = 640;
// 640 threads start with 96 registers each; every warpgroup executes one setmaxnreg, and the budgets must add up to at
// most 5 * 96, or the growing groups never return from theirs.
constexpr int BK1_REGS_LAUNCH = 96, BK1_REGS_ISSUE = 40, BK1_REGS_COMPUTE = 128, BK1_REGS_BUILD = 88;
static_assert(BK1_REGS_ISSUE + 2 * BK1_REGS_COMPUTE + 2 * BK1_REGS_BUILD <= 5 * BK1_REGS_LAUNCH, "register pool must balance");
constexpr int BK1_BUFS = 3;          // S^T / dP^T buffers in TMEM
// A_e / B_e stages.  A stage is released only when the second products of its step have completed, i.e.
// after build -> first products -> P^T/G^T pass -> second products; with two stages the builders (whose
// 32 shared-memory accesses per step take ~1600 cycles next to the tensor cores' operand traffic) waited
// for that chain every step and paced the kernel at ~3000 cycles per step.
constexpr int BK1_STAGES = 3;

enum Bk1Bar {
    BK1_KV_FULL = 0,
    BK1_AB_FULL = 1,     // [BK1_STAGES]
    BK1_AB_EMPTY = 4,    // [BK1_STAGES]
    BK1_S_FULL = 7,      // [BK1_BUFS]
    BK1_P_FULL = 10,     // [BK1_BUFS]
    BK1_G_DONE = 13,     // [BK1_BUFS] second products of the unit have completed
    BK1_DONE = 16,
    BK1_WIN_FREE = 17,   // the builders have finished reading the k2/v2 window of the previous query tile
    BK1_WIN_FULL = 18,   // the window of the current query tile has landed
    BK1_BAR_COUNT = 19
};

enum { ERR_BK1_PRODUCER = 16, ERR_BK1_MMA = 32, ERR_BK1_COMPUTE = 64, ERR_BK1_BUILDER = 128 };

struct BwdParams {
    KernelParams kp;
    float c;        // scale * log2(e)
    int ce;         // CTAs that share a key tile: si x (splits of the offsets)
    int si;         // splits of the (query head, query tile) pairs
    int epc;        // second-key offsets of a CTA
    float *part;    // ce > 1: partial dK1, dV1 [ce][b][nk1][hk][2][d]
    int *status;
};

// padded above half of the SM's shared memory: one CTA per SM, so the 512-column TMEM allocation never waits
constexpr int BK1_WIN_ROWS = 160;    // second-key / second-value rows a query tile can pair with: 32 + 128
inline size_t bk1_smem_bytes() {
    return 1024 + 2 * TILE_BYTES + BK1_STAGES * 2 * TILE_BYTES + 2 * TILE_BYTES + TILE_BYTES + 2 * BK1_WIN_ROWS * 128 + 256;
}

struct Bk1Geom {
    int j0, i_lo, i_hi, n_it, total;
    int e0, e1;     // offsets of this CTA
    int x0, x1;     // its pairs: x = (query head of the group) * n_it + query tile
};

__device__ __forceinline__ int bk1_sweeps(const KernelParams &kp, const Bk1Geom &g, int t) {
    const int last = min(g.i_lo + TQ * t + TQ - 1, g.i_hi);
    return min(g.e1, last + kp.off2 + 1) - g.e0;
}

__device__ __forceinline__ Bk1Geom bk1_geom(const BwdParams &P) {
    const KernelParams &kp = P.kp;
    Bk1Geom g;
    g.j0 = (int)(blockIdx.x / P.ce) * TJ;
    const int split = (int)(blockIdx.x % P.ce), is = split % P.si;
    g.e0 = split / P.si * P.epc;
    g.e1 = min(kp.w2, g.e0 + P.epc);
    // (rows before offset e0's first second key have no work here, so every tile has at least one sweep)
    g.i_lo = max(max(0, g.j0 - kp.off1), g.e0 - kp.off2);
    g.i_hi = min(kp.n - 1, min(g.j0 + TJ - 1, kp.nk1 - 1) + kp.w1 - 1 - kp.off1);
    g.n_it = g.i_hi >= g.i_lo ? (g.i_hi - g.i_lo) / TQ + 1 : 0;
    if (g.e0 >= g.e1) g.n_it = 0;
    g.x0 = g.n_it * kp.g * is / P.si;
    g.x1 = g.n_it * kp.g * (is + 1) / P.si;
    g.total = 0;
    for (int x = g.x0; x < g.x1; ++x) g.total += bk1_sweeps(kp, g, x % g.n_it);
    return g;
}

// ---------------------------------------------------------------- builders (warps 12-19)
// three bf16 terms whose sum is x to fp32 accuracy, packed with five zeros into one 16-byte chunk
__device__ __forceinline__ uint4 split3_bf16(float x) {
    const __nv_bfloat16 h0 = __float2bfloat16_rn(x);
    const float r1 = x - __bfloat162float(h0);
    const __nv_bfloat16 h1 = __float2bfloat16_rn(r1);
    const __nv_bfloat16 h2 = __float2bfloat16_rn(r1 - __bfloat162float(h1));
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    v.x = (uint32_t)__bfloat16_as_ushort(h0) | ((uint32_t)__bfloat16_as_ushort(h1) << 16);
    v.y = (uint32_t)__bfloat16_as_ushort(h2);
    return v;
}

// Head dim 32 leaves half of every 128-byte operand row free: the products q * k2 and dO * v2 are stored as a bf16 value
// (channels 0-31) and its bf16 rest (channels 32-63), which together are exact, and P^T and G^T likewise over the columns of
// S^T and dP^T.  The first products add the rests of A_e / B_e as two more K steps; the second ones take both halves of
// the row as N = 64 columns, whose halves the store adds.  Gradients in bf16 are as far from 64 bits as those of the fp32
// kernels (1.5e-3 to 4.3e-3; 2.9e-3 to 5.9e-3 with rounded operands).  b4 n4096 h8 w512/32: dK1/dV1 1.07 -> 1.64 ms against
// rounded operands, dQ/dK2/dV2 1.33 -> 1.94; 19.7 and 40.0 on the fp32 kernels.
template <int D> constexpr bool bwd_split = D == 32;

template <int D>
__device__ __forceinline__ int bk1_builder(const BwdParams &P, const Bk1Geom &g, const CUtensorMap *mapK2, const CUtensorMap *mapV2,
                                           uint8_t *sAB, uint8_t *sStat, uint8_t *sOnes, uint8_t *sWin,
                                           uint64_t *bars, volatile int *abort_flag) {
    constexpr int NC = D / 16;             // 16-byte chunks of half a row
    const KernelParams &kp = P.kp;
    const int bt = threadIdx.x - 384, r = bt & 127, part = bt >> 7, c0 = part * NC;      // row of the query tile, its half
    const int hk = blockIdx.y, b = blockIdx.z;
    const __nv_bfloat16 *q = reinterpret_cast<const __nv_bfloat16 *>(kp.q.p);
    const __nv_bfloat16 *k2 = reinterpret_cast<const __nv_bfloat16 *>(kp.k2.p);
    const __nv_bfloat16 *dout = reinterpret_cast<const __nv_bfloat16 *>(kp.dout.p);
    const __nv_bfloat16 *v2 = reinterpret_cast<const __nv_bfloat16 *>(kp.v2.p);
    // the constant key-side tile: three ones per row (one per term of the split statistics)
    if (part == 0) {
        uint4 one = make_uint4(0x3f803f80u, 0x00003f80u, 0u, 0u);
#pragma unroll
        for (int cc = 0; cc < 8; ++cc)
            *reinterpret_cast<uint4 *>(sOnes + sw128_offset(r, cc)) = cc == 0 ? one : make_uint4(0u, 0u, 0u, 0u);
    }
    const float inv_c = 1.f / P.c;
    int s = 0, tile_counter = 0;
    for (int x = g.x0; x < g.x1; ++x, ++tile_counter) {
        const int t = x % g.n_it, h = hk * kp.g + x / g.n_it;
        const int i = g.i_lo + TQ * t + r;
        const bool iv = i <= g.i_hi;
        const int ne = bk1_sweeps(kp, g, t);
        // The k2 / v2 rows this query tile pairs with over all sweeps (positions it0 - e0 - 32 .. it0 - e0 + 127)
        // are staged once per tile by TMA; every step then reads its rows from shared memory.
        const bool win = P.epc <= 32;
        if (win) {
            if (tile_counter > 0) mbar_arrive(&bars[BK1_WIN_FREE]);
            if (bt == 0) {
                if (tile_counter > 0 && !mbar_wait(&bars[BK1_WIN_FREE], (tile_counter - 1) & 1, abort_flag)) return ERR_BK1_BUILDER;
                mbar_arrive_expect_tx(&bars[BK1_WIN_FULL], 2 * BK1_WIN_ROWS * 128);
                const int row0 = g.i_lo + TQ * t + kp.off2 - g.e0 - 32;
                for (int bx = 0; bx < BK1_WIN_ROWS / 32; ++bx) {
                    tma_load_4d(sWin + bx * 4096, mapK2, &bars[BK1_WIN_FULL], 0, hk, row0 + 32 * bx, b);
                    tma_load_4d(sWin + BK1_WIN_ROWS * 128 + bx * 4096, mapV2, &bars[BK1_WIN_FULL], 0, hk, row0 + 32 * bx, b);
                }
            }
            if (!mbar_wait(&bars[BK1_WIN_FULL], tile_counter & 1, abort_flag, 64, 1)) return ERR_BK1_BUILDER;
        }
        uint4 qv[NC], dv[NC];
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) { qv[cc] = make_uint4(0, 0, 0, 0); dv[cc] = make_uint4(0, 0, 0, 0); }
        float stat = 0.f;                   // half 0: -lse2 / c, half 1: -D
        if (iv) {
            const __nv_bfloat16 *qp = q + elem_off(kp.q, b, i, h) + c0 * 8;
            const __nv_bfloat16 *dp = dout + elem_off(kp.dout, b, i, h) + c0 * 8;
#pragma unroll
            for (int cc = 0; cc < NC; ++cc) {
                qv[cc] = *reinterpret_cast<const uint4 *>(qp + cc * 8);
                dv[cc] = *reinterpret_cast<const uint4 *>(dp + cc * 8);
            }
            const int64_t o = ((int64_t)b * kp.hq + h) * kp.n + i;
            stat = part == 0 ? -kp.lse[o] * 1.4426950408889634f * inv_c : -kp.delta[o];
        }
        for (int e = 0; e < ne; ++e, ++s) {
            const int stage = s % BK1_STAGES;
            if (s >= BK1_STAGES && !warp_wait(&bars[BK1_AB_EMPTY + stage], (s / BK1_STAGES - 1) & 1, abort_flag, 2)) return ERR_BK1_BUILDER;
            if (e == 0) {
                // Statistics of this query tile: two K = 16 slabs (-lse2/c, -D) of a four-slab tile; two
                // such tiles hold the last four query tiles.  Step s - 3 has completed, and every tile has
                // at least one step, so the slabs of four tiles ago are no longer read.
                uint8_t *st = sStat + (size_t)((tile_counter >> 1) & 1) * TILE_BYTES;
                const int ch = (tile_counter & 1) * 4 + 2 * part;
                *reinterpret_cast<uint4 *>(st + sw128_offset(r, ch)) = split3_bf16(stat);
                *reinterpret_cast<uint4 *>(st + sw128_offset(r, ch + 1)) = make_uint4(0u, 0u, 0u, 0u);
            }
            uint8_t *dA = sAB + (size_t)stage * 2 * TILE_BYTES;
            uint8_t *dB = dA + TILE_BYTES;
            const int kk = i + kp.off2 - g.e0 - e;
            const bool ok = iv && kk >= 0;
            const __nv_bfloat16 *kp2 = k2 + elem_off(kp.k2, b, ok ? kk : 0, hk) + c0 * 8;
            const __nv_bfloat16 *vp2 = v2 + elem_off(kp.v2, b, ok ? kk : 0, hk) + c0 * 8;
            const int wr = r + 32 - e;                       // row of the staged window
            const uint8_t *wk = sWin + wr * 128, *wv = wk + BK1_WIN_ROWS * 128;
#pragma unroll
            for (int cc = 0; cc < NC; ++cc) {
                uint4 a = make_uint4(0, 0, 0, 0), bb = make_uint4(0, 0, 0, 0), ar = a, br = a;
                if (ok) {
                    const uint4 kv = win ? *reinterpret_cast<const uint4 *>(wk + (((c0 + cc) ^ (wr & 7)) << 4))
                                         : *reinterpret_cast<const uint4 *>(kp2 + cc * 8);
                    const uint4 vv = win ? *reinterpret_cast<const uint4 *>(wv + (((c0 + cc) ^ (wr & 7)) << 4))
                                         : *reinterpret_cast<const uint4 *>(vp2 + cc * 8);
                    a.x = mul_bf16x2(qv[cc].x, kv.x); a.y = mul_bf16x2(qv[cc].y, kv.y);
                    a.z = mul_bf16x2(qv[cc].z, kv.z); a.w = mul_bf16x2(qv[cc].w, kv.w);
                    bb.x = mul_bf16x2(dv[cc].x, vv.x); bb.y = mul_bf16x2(dv[cc].y, vv.y);
                    bb.z = mul_bf16x2(dv[cc].z, vv.z); bb.w = mul_bf16x2(dv[cc].w, vv.w);
                    if constexpr (bwd_split<D>) { ar = mul_rest_bf16x8(qv[cc], kv, a); br = mul_rest_bf16x8(dv[cc], vv, bb); }
                }
                *reinterpret_cast<uint4 *>(dA + sw128_offset(r, c0 + cc)) = a;
                *reinterpret_cast<uint4 *>(dB + sw128_offset(r, c0 + cc)) = bb;
                if constexpr (bwd_split<D>) {
                    *reinterpret_cast<uint4 *>(dA + sw128_offset(r, 4 + c0 + cc)) = ar;
                    *reinterpret_cast<uint4 *>(dB + sw128_offset(r, 4 + c0 + cc)) = br;
                }
            }
            fence_proxy_async_smem();
            mbar_arrive(&bars[BK1_AB_FULL + stage]);
        }
    }
    return 0;
}

// ---------------------------------------------------------------- issuers of S^T (warp 1) and dP^T (warp 2)
// Unit u is half u & 1 of step u / 2 and uses buffer u % 3.  which = 0: S^T = K1 A_e^T - lse2 / c; 1: dP^T = V1 B_e^T - D.
template <int D>
__device__ __forceinline__ int bk1_mma_first(const KernelParams &kp, const Bk1Geom &g, int which, uint32_t tmem, uint8_t *sKV,
                                             uint8_t *sAB, uint8_t *sStat, uint8_t *sOnes, uint64_t *bars, volatile int *abort_flag) {
    constexpr uint32_t IDESC_F = idesc_bf16(128, 64, false, false);
    const uint64_t dT = smem_desc_sw128(smem_u32(sKV));
    const uint64_t dAB = smem_desc_sw128(smem_u32(sAB + which * TILE_BYTES));
    const uint64_t dSt = smem_desc_sw128(smem_u32(sStat)), dOnes = smem_desc_sw128(smem_u32(sOnes));
    if (!mbar_wait_warp(&bars[BK1_KV_FULL], 0, abort_flag)) return ERR_BK1_MMA;
    int s = 0, tile_counter = 0, buf = 0, use = 0;
    for (int x = g.x0; x < g.x1; ++x, ++tile_counter) {
        const int t = x % g.n_it;
        const int ne = bk1_sweeps(kp, g, t);
        // slab (16 channels = 32 bytes = 2 descriptor units) of the statistics tile that holds this query tile
        const uint64_t stL0 = dSt + (uint64_t)((((tile_counter >> 1) & 1) * TILE_BYTES) >> 4) + (uint64_t)((tile_counter & 1) * 4);
        for (int e = 0; e < ne; ++e, ++s) {
            const int stage = s % BK1_STAGES;
            if (!mbar_wait_warp(&bars[BK1_AB_FULL + stage], (s / BK1_STAGES) & 1, abort_flag, 0, 1)) return ERR_BK1_MMA;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                // the buffer holds P^T / G^T of its last unit until the second products of that unit are done
                if (use >= 1 && !mbar_wait_warp(&bars[BK1_G_DONE + buf], (use - 1) & 1, abort_flag, 0, 2)) return ERR_BK1_MMA;
                tc_fence_after();
                const uint64_t a = dAB + (uint64_t)((stage * 2 * TILE_BYTES + half * 8192) >> 4);
                const uint64_t st = stL0 + (uint64_t)((half * 8192) >> 4) + (uint64_t)(which * 2);
                const uint32_t d = tmem + buf * 128 + which * 64;
                if (elect_one()) {
#pragma unroll
                for (int k = 0; k < D / 16; ++k) mma_ss(d, dT + 2 * k, a + 2 * k, IDESC_F, k > 0 ? 1u : 0u);
                if constexpr (bwd_split<D>) {
#pragma unroll
                    for (int k = 0; k < D / 16; ++k) mma_ss(d, dT + 2 * k, a + 4 + 2 * k, IDESC_F, 1u);
                }
                mma_ss(d, dOnes, st, IDESC_F, 1u);                // - lse2_i / c, or - D_i
                tc_commit(&bars[BK1_S_FULL + buf]);
                }
                if (++buf == BK1_BUFS) { buf = 0; ++use; }
            }
        }
    }
    return 0;
}

// ---------------------------------------------------------------- issuer of dV1, dK1 (warp 0)
template <int D>
__device__ __forceinline__ int bk1_mma_second(const Bk1Geom &g, uint32_t tmem, uint8_t *sAB, uint64_t *bars, volatile int *abort_flag) {
    constexpr bool SPLIT = bwd_split<D>;
    constexpr uint32_t IDESC_G = idesc_bf16(128, SPLIT ? 2 * D : D, false, true);    // B operand MN-major
    // P^T / G^T of keys [16 k, +16): side by side, or with their rests behind every 32 keys
    auto cols = [](int k) { return SPLIT ? (k >> 1) * 32 + (k & 1) * 8 : 8 * k; };
    const uint64_t dAB = smem_desc_sw128(smem_u32(sAB));
    int buf = 0, use = 0;
    for (int s = 0; s < g.total; ++s) {
        const int stage = s % BK1_STAGES;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            if (!mbar_wait_warp(&bars[BK1_P_FULL + buf], use & 1, abort_flag, 0, 1)) return ERR_BK1_MMA;
            tc_fence_after();
            const uint64_t a = dAB + (uint64_t)((stage * 2 * TILE_BYTES + half * 8192) >> 4), bq = a + (TILE_BYTES >> 4);
            const uint32_t tp = tmem + buf * 128, tg = tp + 64;
            const uint32_t first = (s > 0 || half > 0) ? 1u : 0u;
            if (elect_one()) {
#pragma unroll
            for (int k = 0; k < 4; ++k) mma_ts(tmem + 448, tp + cols(k), bq + 128 * k, IDESC_G, k > 0 ? 1u : first);
#pragma unroll
            for (int k = 0; k < 4; ++k) mma_ts(tmem + 384, tg + cols(k), a + 128 * k, IDESC_G, k > 0 ? 1u : first);
            if constexpr (SPLIT) {
#pragma unroll
                for (int k = 0; k < 4; ++k) mma_ts(tmem + 448, tp + 16 + cols(k), bq + 128 * k, IDESC_G, 1u);
#pragma unroll
                for (int k = 0; k < 4; ++k) mma_ts(tmem + 384, tg + 16 + cols(k), a + 128 * k, IDESC_G, 1u);
            }
            tc_commit(&bars[BK1_G_DONE + buf]);
            if (half == 1) tc_commit(&bars[BK1_AB_EMPTY + stage]);
            }
            if (++buf == BK1_BUFS) { buf = 0; ++use; }
        }
    }
    if (elect_one()) tc_commit(&bars[BK1_DONE]);
    return 0;
}

// ---------------------------------------------------------------- compute (group h: units of half h; warps 4-7, 8-11)
template <int D>
__device__ __forceinline__ int bk1_compute(const BwdParams &P, const Bk1Geom &g, int half, uint32_t tmem,
                                           uint64_t *bars, volatile int *abort_flag) {
    const KernelParams &kp = P.kp;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = (warp & 3) * 32 + lane;          // key row within the tile = TMEM lane
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int hk = blockIdx.y, b = blockIdx.z;
    const int j = g.j0 + r;
    const bool jv = j < kp.nk1;
    const uint64_t c2 = f2_pack(P.c, P.c);

    // the walk over the steps; a wait that runs out ends it early, the rows are then reported as NaN below
    auto walk = [&]() -> int {
        int s = 0, u = half;
        for (int xt = g.x0; xt < g.x1; ++xt) {
            const int t = xt % g.n_it;
            const int it0 = g.i_lo + TQ * t;
            const int ne = bk1_sweeps(kp, g, t);
            const int base = j - kp.off1 - it0;                       // column of the diagonal i + off1 == j
            const int hi = (jv ? min(min(TQ - 1, base + kp.w1 - 1), g.i_hi - it0) : -1) - half * 64;
            for (int e = 0; e < ne; ++e, ++s, u += 2) {
                const uint32_t buf = lane_addr + (u % BK1_BUFS) * 128;
                const int lo = max(max(0, base), g.e0 + e - kp.off2 - it0) - half * 64;     // valid columns: lo <= col <= hi
                if (!warp_wait(&bars[BK1_S_FULL + u % BK1_BUFS], (u / BK1_BUFS) & 1, abort_flag, 1)) return ERR_BK1_COMPUTE;
                tc_fence_after();
                const bool full = __all_sync(0xffffffffu, lo <= 0 && hi >= 63);
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    constexpr bool SPLIT = bwd_split<D>;
                    uint32_t sv[32], dv[32], pk[16], gk[16], pr[SPLIT ? 16 : 1], gr[SPLIT ? 16 : 1];
                    tmem_ld32(buf + ch * 32, sv);
                    tmem_ld32(buf + 64 + ch * 32, dv);
                    tmem_wait_ld(sv);
                    tmem_waited(dv);
                    // the accumulators already hold S^T - lse2 / c and dP^T - D
                    auto pair = [&](int x, float a0, float a1) {
                        const float p0 = ex2(a0), p1 = ex2(a1);
                        float g0, g1;
                        f2_unpack(f2_mul(f2_pack(p0, p1), f2_pack(dv[x], dv[x + 1])), g0, g1);
                        pk[x >> 1] = pack_bf16(p0, p1);
                        gk[x >> 1] = pack_bf16(g0, g1);
                        if constexpr (SPLIT) {
                            pr[x >> 1] = pack_rest(p0, p1, pk[x >> 1]);
                            gr[x >> 1] = pack_rest(g0, g1, gk[x >> 1]);
                        }
                    };
                    if (full) {
#pragma unroll
                        for (int x = 0; x < 32; x += 2) {
                            float a0, a1;
                            f2_unpack(f2_mul(f2_pack(sv[x], sv[x + 1]), c2), a0, a1);
                            pair(x, a0, a1);
                        }
                    } else {
                        // valid columns are the integers in [lo, hi]: 2048 (half + 1/2 - |col - mid|) is at least 1024
                        // inside and at most -1024 outside, so the minimum with it leaves the exponents of valid cells
                        // alone and makes P exactly 0 elsewhere, whatever S is there (FMA pipe instead of compares and
                        // selects on the ALU pipe; all values are exact)
                        const float mid = 1024.f * (float)(lo + hi) - 2048.f * (float)(ch * 32), half_w = 1024.f * (float)(hi - lo + 1);
#pragma unroll
                        for (int x = 0; x < 32; x += 2) {
                            float a0, a1;
                            f2_unpack(f2_mul(f2_pack(sv[x], sv[x + 1]), c2), a0, a1);
                            pair(x, fminf(a0, half_w - fabsf(2048.f * x - mid)), fminf(a1, half_w - fabsf(2048.f * (x + 1) - mid)));
                        }
                    }
                    // over columns of S^T / dP^T that this thread has already read
                    if constexpr (SPLIT) {
                        tmem_st16(buf + ch * 32, pk);
                        tmem_st16(buf + ch * 32 + 16, pr);
                        tmem_st16(buf + 64 + ch * 32, gk);
                        tmem_st16(buf + 64 + ch * 32 + 16, gr);
                    } else {
                        tmem_st16(buf + ch * 16, pk);
                        tmem_st16(buf + 64 + ch * 16, gk);
                    }
                }
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(&bars[BK1_P_FULL + u % BK1_BUFS]);
            }
        }
        return 0;
    };
    int err = walk();
    // drain: group 0 writes dK1, group 1 writes dV1
    if (err == 0 && !warp_wait(&bars[BK1_DONE], 0, abort_flag)) err = ERR_BK1_COMPUTE;
    const bool bad = __any_sync(0xffffffffu, err != 0) || *abort_flag != 0;
    tc_fence_after();
    const bool gbf16 = kp.grad_bf16 != 0;
    const TensorRef &dst = half == 0 ? kp.dk1 : kp.dv1;
    const float mul = half == 0 ? kp.scale : 1.f;
#pragma unroll 1
    for (int hf = 0; hf < D / 32; ++hf) {
        uint32_t w[32];
        tmem_ld32(lane_addr + 384 + half * 64 + hf * 32, w);
        tmem_wait_ld(w);
        if constexpr (bwd_split<D>) {
            uint32_t rest[32];
            tmem_ld32(lane_addr + 384 + half * 64 + 32, rest);
            tmem_wait_ld(rest);
#pragma unroll
            for (int x = 0; x < 32; ++x) w[x] = __float_as_uint(__uint_as_float(w[x]) + __uint_as_float(rest[x]));
        }
        if (P.ce > 1 && jv) {
            float *row = P.part + (((((size_t)(blockIdx.x % P.ce) * kp.b + b) * kp.nk1 + j) * kp.hk + hk) * 2 + half) * D + hf * 32;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                float4 x;
                x.x = __uint_as_float(w[u * 4]); x.y = __uint_as_float(w[u * 4 + 1]);
                x.z = __uint_as_float(w[u * 4 + 2]); x.w = __uint_as_float(w[u * 4 + 3]);
                if (g.total == 0) x = make_float4(0.f, 0.f, 0.f, 0.f);
                if (bad) x = make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F);
                *reinterpret_cast<float4 *>(row + u * 4) = x;
            }
        } else if (jv) {
            const int64_t off = elem_off(dst, b, j, hk) + hf * 32;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                float x[4];
#pragma unroll
                for (int z = 0; z < 4; ++z) x[z] = bad ? CUDART_NAN_F : (g.total > 0 ? __uint_as_float(w[u * 4 + z]) : 0.f) * mul;
                store_vec<4>(dst.p, off + u * 4, gbf16, x);
            }
        }
    }
    return err;
}

template <int D>
__global__ void __launch_bounds__(BK1_THREADS, 1)
bwd_k1_kernel(const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapV,
              const __grid_constant__ CUtensorMap mapK2, const __grid_constant__ CUtensorMap mapV2, const BwdParams P) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = align_smem(smem_raw);
    uint8_t *sK = smem;
    uint8_t *sV = sK + TILE_BYTES;
    uint8_t *sAB = sV + TILE_BYTES;                       // BK1_STAGES x (A tile, B tile)
    uint8_t *sStat = sAB + BK1_STAGES * 2 * TILE_BYTES;   // 2 tiles x 2 query tiles x (-lse2/c slab, -D slab)
    uint8_t *sOnes = sStat + 2 * TILE_BYTES;              // constant: three ones per row
    uint8_t *sWin = sOnes + TILE_BYTES;                   // staged k2 rows, then v2 rows (160 x 128 B each)
    uint64_t *bars = reinterpret_cast<uint64_t *>(sWin + 2 * BK1_WIN_ROWS * 128);
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bars + BK1_BAR_COUNT);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_holder + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);       // warp-uniform, and known to be
    if (threadIdx.x == 0) {
        for (int x = 0; x < BK1_BAR_COUNT; ++x) {
            uint32_t count = 1;
            if ((x >= BK1_AB_FULL && x < BK1_AB_FULL + BK1_STAGES) || x == BK1_WIN_FREE) count = 256;     // every builder
            else if (x >= BK1_P_FULL && x < BK1_P_FULL + BK1_BUFS) count = 128;
            else if (x >= BK1_S_FULL && x < BK1_S_FULL + BK1_BUFS) count = 2;        // one commit from each first-product issuer
            mbar_init(&bars[x], count);
        }
        *abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_holder, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_holder;
    const Bk1Geom g = bk1_geom(P);

    int err = 0;
#ifdef SA2_PROF
    const long long prof_t0 = clock64();
    sa2::sm100::prof_begin();
#endif
    if (warp < 4) {
        reg_dealloc<BK1_REGS_ISSUE>();
        if (warp == 0) {
            if (g.total > 0) {
                if (elect_one()) {
                    prefetch_tmap(&mapK);
                    prefetch_tmap(&mapV);
                    mbar_arrive_expect_tx(&bars[BK1_KV_FULL], 2 * TILE_BYTES);
                    tma_load_4d(sK, &mapK, &bars[BK1_KV_FULL], 0, blockIdx.y, g.j0, blockIdx.z);
                    tma_load_4d(sV, &mapV, &bars[BK1_KV_FULL], 0, blockIdx.y, g.j0, blockIdx.z);
                }
                err = bk1_mma_second<D>(g, tmem, sAB, bars, abort_flag);
                // the tile must have landed before the CTA may exit, even if every other role gave up
                if (!mbar_wait_warp(&bars[BK1_KV_FULL], 0, abort_flag)) err |= ERR_BK1_PRODUCER;
            } else if (elect_one()) {
                tc_commit(&bars[BK1_DONE]);
            }
        } else if (warp == 1) {
            if (g.total > 0) err = bk1_mma_first<D>(P.kp, g, 0, tmem, sK, sAB, sStat, sOnes, bars, abort_flag);
        } else if (warp == 2) {
            if (g.total > 0) err = bk1_mma_first<D>(P.kp, g, 1, tmem, sV, sAB, sStat, sOnes, bars, abort_flag);
        }
    } else if (warp < 12) {
        reg_alloc<BK1_REGS_COMPUTE>();
        err = bk1_compute<D>(P, g, (warp - 4) >> 2, tmem, bars, abort_flag);
    } else {
        reg_dealloc<BK1_REGS_BUILD>();
        err = bk1_builder<D>(P, g, &mapK2, &mapV2, sAB, sStat, sOnes, sWin, bars, abort_flag);
    }
    if (err) atomicOr(P.status, err);
    SA2_PROF_ADD(0, clock64() - prof_t0);
    SA2_PROF_END();

    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// ------------------------------------------------------------------ host side
// What the split rules look at besides the (clamped) shape.
struct BwdCaller {
    int w2;        // the caller's second window, however short the sequence
    int batch;     // batch elements of the whole call: a part of it (sa2_bwd_part) is cut as the whole is, for the same bits
};
// Cycles of `batch` times `ctas` CTAs of `one` cycles each: whole waves of one CTA per SM.
// A rule for one and for eight elements at once, which needed no batch, cost many short sequences dear: with eight ranges
// of offsets in both kernels b128 n128 h8 d64 w512/32 took 2506 us and 2.0 GiB of scratch, 988 us and 80 MiB with one.
// A split must promise 8 %: at 7 % b2 n4096 h8 d64 w512/32 (3.5 waves of CTAs into 6.9 shorter ones) got 5 % slower.
constexpr double SPLIT_GAIN = 0.92;
inline double split_cost(int64_t ctas, double one, int batch, int sms) { return (double)((ctas * batch + sms - 1) / sms) * one; }
// CTAs per key tile: splits of the (query head, query tile) pairs first, then of the offsets.  A CTA costs ~8000 cycles
// of set-up, loads and store, a pair ~4000 (its rows and second-key window), a step of 128 query rows and one offset
// ~2600 (twice that at head dim 128), measured on a B200; twice as much again with more than 32 offsets, whose second keys
// do not fit the staged window (b5 n1500 hq16 hk2 d128 w700/40 with 40 offsets per CTA 5441 us, with 5 of them 2815).
struct K1Split { int si, se, epc; };
inline K1Split k1_split(const sa2_shape &s, const BwdCaller &call, int sms) {
    const int nk1 = s.n + s.off1, rows = s.w1 + TJ - 1 < s.n ? s.w1 + TJ - 1 : s.n;
    const int64_t tiles = (int64_t)((nk1 + TJ - 1) / TJ) * s.hk;
    const int pairs = (s.hq / s.hk) * ((rows + TQ - 1) / TQ), w2 = s.w2 < s.n + s.off2 ? s.w2 : s.n + s.off2;
    const double step = s.d == 128 ? 5200. : 2600.;
    K1Split best{1, 1, w2};
    double best_cost = 0.;
    for (int se = 1; se <= 16 && se <= w2; ++se)
        for (int si = 1; si * se <= 16 && si <= pairs; ++si) {
            const int epc = (w2 + se - 1) / se;
            const double cost = split_cost(tiles * si * se, 8000. + (pairs + si - 1) / si * (4000. + epc * (epc > 32 ? 2. : 1.) * step), call.batch, sms);
            if (best_cost == 0. || cost < SPLIT_GAIN * best_cost) { best = K1Split{si, (w2 + epc - 1) / epc, epc}; best_cost = cost; }
        }
    return best;
}
inline size_t k1_part_bytes(const sa2_shape &s, int ce) {
    return ce == 1 ? 0 : (size_t)ce * s.b * (s.n + s.off1) * s.hk * 2 * s.d * sizeof(float);
}

}  // namespace tc
}  // namespace sa2
