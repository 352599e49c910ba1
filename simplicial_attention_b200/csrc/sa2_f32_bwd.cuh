// Backward of fp32 tensors on tcgen05 tensor cores, head dims 32 and 64 (operands of three bf16 terms, sa2_f32_common.cuh).
//
// One kernel body in two modes, each with 128 key rows as the rows of its logit tiles and units of 64 columns:
//   MODE_K1: rows are first keys j, columns are query rows i of one offset e;   A_e, B_e are rebuilt for every unit
//       S^T = K1 A_e^T   dP^T = V1 B_e^T      dK1 += G^T A_e      dV1 += P^T B_e
//   MODE_K2: rows are second keys k (with the query i = k + e), columns are first keys; A_e, B_e stay for a sweep of units
//       S = A_e K1^T     dP = B_e V1^T        U = G K1   W = P V1
//       at the end of a sweep   dK2_k += U q_{k+e}   dV2_k += W dO_{k+e}   dQ_{k+e} += U k2_k
//   with A_e = scale log2(e) q_i * k2_{i-e}, B_e = dO_i * v2_{i-e}, P = exp2(S - lse), G = P (dP - D).
// So the sums that last (dK1, dV1; dK2, dV2) belong to a row of the tile, live in registers over all offsets and query heads
// of the group and need no atomics.  dQ rows move by one row a sweep: a ring of 128 rows in shared memory, whose finished row
// goes to a slab of 127 + epc rows in scratch; the reduction adds the slabs of the tiles and offset ranges in order.
//
// Warps (512 threads, 640 in MODE_K2): 0 / 3 issuers of U / W, 1 / 2 of S / dP; then one or two groups of four that form P and G, four
// that build A_e (K1) and sum U, four that build B_e (V1) and sum W.  TMEM: buffer x: S, then the terms of P [192 x, +96), dP and G
// [192 x + 96, +96); U [384, +64), W [448, +64).
//
// Bound: a unit's 96 products fetch 384 KB from shared memory, ~3100 cycles; the chain operands -> S / dP -> P / G -> U / W of two
// units in flight takes ~6000 cycles a unit.  b1 n1024 h8 d64 w512/32: 5.5 ms on the scalar kernels -> 0.54 (MODE_K1) + 0.60 ms;
// forward + backward 7.5 -> 1.45 ms, b1 n128 h2 d32 full causal 0.30 -> 0.10 ms.
#pragma once
#include "sa2_f32_common.cuh"
#include "sa2_tc_bwd_k1.cuh"

namespace sa2 {
namespace f32 {

enum { MODE_K1 = 0, MODE_K2 = 1 };
// Compute groups: two in MODE_K2, 32 columns of a unit each (0.63 -> 0.60 ms on b1 n1024 h8 d64 w512/32), one in MODE_K1 (0.53; 0.63
// with two, whose registers the sums and the rows of q would have to give).
template <int MODE> struct BwdCfg {
    static constexpr int GROUPS = MODE == MODE_K1 ? 1 : 2, THREADS = 384 + 128 * GROUPS;
    static constexpr int REGS_LAUNCH = GROUPS == 2 ? 96 : 128, REGS_ISSUE = GROUPS == 2 ? 32 : 40, REGS_COMPUTE = GROUPS == 2 ? 80 : 152;
    static constexpr int REGS_SUM = GROUPS == 2 ? 144 : 160;
    static_assert(REGS_ISSUE + GROUPS * REGS_COMPUTE + 2 * REGS_SUM == THREADS / 128 * REGS_LAUNCH, "register pool must balance");
};

enum BwdBar {
    B_M_FULL = 0,      // [2] row-side operand of S / dP
    B_M_EMPTY = 2,     // [2]
    B_N_FULL = 4,      // [2 operands][2 slots] column-side operands
    B_S_FULL = 8,      // [2 buffers] S and dP
    B_P_FULL = 10,     // [2 buffers] terms of P and G
    B_DONE = 12,       // [2: U, W][2 buffers] the second product of the unit
    B_ACC_EMPTY = 16,  // [2: U, W]
    B_RING = 18,       // the sweep is in the dQ ring
    B_BAR_COUNT = 19
};

struct BwdParams {
    KernelParams kp;
    int nsplit;        // CTAs that share a tile: head (MODE_K1: head and query unit) splits x offset splits
    int hsplit;
    int epc;           // offsets of a CTA
    int tiles;         // MODE_K2: tiles of a head
    float *part;       // partial dK, dV [nsplit][b][rows][hk][2][d], if nsplit > 1
    float *slab;       // MODE_K2: dQ [b][hq][tiles][offset splits][127 + epc][d]
    int *redo;         // [b]: set where the scalar kernels have to do the mode's gradients
    int *status;
};

template <int D, int MODE> inline size_t bwd_smem_bytes() {
    return 1024 + 2 * Planes<D>::bytes(ROWS) + 4 * Planes<D>::bytes(UNIT) + (MODE == MODE_K2 ? ROWS * D * 4 : 2 * UNIT * 8) + 256;
}

// The units of a CTA, one after the other.
//   MODE_K2: for every query head, every offset, the 64-key units its rows see
//   MODE_K1: for every (query head, 64-row query unit), every offset: one unit
template <int MODE> struct Walk {
    const KernelParams &kp;
    int r0, hk;                     // first row of the tile
    int x, x1;                      // K1: pairs of (query head of the group) * n_it + query unit; K2: query heads
    int e, ea, eb;                  // offset; K2: the offsets [ea, eb] that have rows
    int c0, w, nw;                  // first column of the unit (key or query row); K2: unit of the sweep
    int i_lo, i_hi, n_it, e0, e1;

    __device__ __forceinline__ Walk(const BwdParams &P) : kp(P.kp) {
        const int split = (int)blockIdx.x % P.nsplit, hs = split % P.hsplit;
        r0 = (int)blockIdx.x / P.nsplit * ROWS;
        hk = blockIdx.y;
        e0 = split / P.hsplit * P.epc;
        e1 = min(kp.w2, e0 + P.epc);
        if constexpr (MODE == MODE_K2) {
            const int top = min(r0 + ROWS, kp.nk2) - 1;
            ea = max(e0, kp.off2 - top);
            eb = min(e1 - 1, kp.n - 1 + kp.off2 - r0);
            x = kp.g * hs / P.hsplit;
            x1 = ea <= eb ? kp.g * (hs + 1) / P.hsplit : x;
            e = ea;
            if (!done()) sweep();
        } else {
            const int top = min(r0 + ROWS, kp.nk1) - 1;
            i_lo = max(max(0, r0 - kp.off1), e0 - kp.off2);
            i_hi = min(kp.n - 1, top + kp.w1 - 1 - kp.off1);
            n_it = e0 < e1 && i_hi >= i_lo ? (i_hi - i_lo) / UNIT + 1 : 0;
            x = n_it * kp.g * hs / P.hsplit;
            x1 = n_it * kp.g * (hs + 1) / P.hsplit;
            if (!done()) sweep();
        }
    }
    __device__ __forceinline__ bool done() const { return x >= x1; }
    __device__ __forceinline__ int head() const { return hk * kp.g + (MODE == MODE_K2 ? x : x / n_it); }
    __device__ __forceinline__ bool first() const { return MODE == MODE_K2 ? w == 0 : e == e0; }
    __device__ __forceinline__ bool last() const { return MODE == MODE_K2 ? w + 1 == nw : e == eb; }
    __device__ __forceinline__ void sweep() {
        if constexpr (MODE == MODE_K2) {
            const int base = r0 - kp.off2 + e;                      // query row of the tile's first row
            const int lo = max(0, base), hi = min(kp.n - 1, min(base + ROWS, kp.nk2 - kp.off2 + e) - 1);
            c0 = max(0, lo + kp.off1 - kp.w1 + 1);
            w = 0;
            nw = (hi + kp.off1 - c0) / UNIT + 1;
        } else {
            c0 = i_lo + UNIT * (x % n_it);
            e = e0;
            eb = min(e1, min(c0 + UNIT - 1, i_hi) + kp.off2 + 1) - 1;      // at least e0
        }
    }
    __device__ __forceinline__ void next() {
        if constexpr (MODE == MODE_K2) {
            c0 += UNIT;
            if (++w < nw) return;
            if (++e > eb) { e = ea; ++x; }
            if (!done()) sweep();
        } else {
            if (++e <= eb) return;
            ++x;
            if (!done()) sweep();
        }
    }
};

// S = M N^T (which = 0) or dP (1)
template <int D, int MODE>
__device__ __forceinline__ int bwd_first(const BwdParams &P, int which, uint32_t tmem, const uint8_t *sM, const uint8_t *sN, uint64_t *bars,
                                         volatile int *abort_flag) {
    const uint64_t dM = smem_desc_sw128(smem_u32(sM) + which * Planes<D>::bytes(ROWS));
    const uint64_t dN = smem_desc_sw128(smem_u32(sN) + which * 2 * Planes<D>::bytes(UNIT));
    int u = 0, s = 0;
    for (Walk<MODE> wk(P); !wk.done(); wk.next(), ++u) {
        const int buf = u & 1;
        if ((MODE == MODE_K2 ? wk.first() : u == 0) && !mbar_wait_warp(&bars[B_M_FULL + which], s++ & 1, abort_flag, 0, 1)) return ERR_BWD;
        if (!mbar_wait_warp(&bars[B_N_FULL + 2 * which + buf], (u >> 1) & 1, abort_flag, 0, 2)) return ERR_BWD;
        // the columns of S hold the terms of P until W of their unit is done, those of dP the terms of G until U is
        if (u >= 2 && !mbar_wait_warp(&bars[B_DONE + 2 * (1 - which) + buf], ((u >> 1) - 1) & 1, abort_flag, 0, 3)) return ERR_BWD;
        tc_fence_after();
        if (elect_one()) {
            issue_nt<D, MODE == MODE_K1>(tmem + 192 * buf + 96 * which + LOGITS, dM, dN + buf * (Planes<D>::bytes(UNIT) >> 4));
            tc_commit(&bars[B_S_FULL + buf]);
            if (MODE == MODE_K2 && wk.last()) tc_commit(&bars[B_M_EMPTY + which]);
        }
    }
    return 0;
}
// U = G N (which = 0) or W = P N (1)
template <int D, int MODE>
__device__ __forceinline__ int bwd_second(const BwdParams &P, int which, uint32_t tmem, const uint8_t *sN, uint64_t *bars, volatile int *abort_flag) {
    const uint64_t dN = smem_desc_sw128(smem_u32(sN) + which * 2 * Planes<D>::bytes(UNIT));
    int u = 0;
    for (Walk<MODE> wk(P); !wk.done(); wk.next(), ++u) {
        const int buf = u & 1;
        if (!mbar_wait_warp(&bars[B_P_FULL + buf], (u >> 1) & 1, abort_flag, 0, 1)) return ERR_BWD;
        if (u >= 1 && !mbar_wait_warp(&bars[B_ACC_EMPTY + which], (u - 1) & 1, abort_flag, 0, 2)) return ERR_BWD;
        tc_fence_after();
        if (elect_one()) {
            issue_pv<D>(tmem + 384 + 64 * which, tmem + 192 * buf + 96 * (1 - which), dN + buf * (Planes<D>::bytes(UNIT) >> 4));
            tc_commit(&bars[B_DONE + 2 * which + buf]);
        }
    }
    return 0;
}

// P and G of every unit, a thread per row; group cg of the compute groups
template <int D, int MODE>
__device__ __forceinline__ int bwd_compute(const BwdParams &P, int cg, uint32_t tmem, const float2 *stats, uint64_t *bars, volatile int *abort_flag) {
    const KernelParams &kp = P.kp;
    const int r = threadIdx.x & 127, b = blockIdx.z;
    const uint32_t lanes = tmem + ((uint32_t)(r & 96) << 16);
    float lse2 = 0.f, dl = 0.f;
    int u = 0;
    for (Walk<MODE> wk(P); !wk.done(); wk.next(), ++u) {
        const int buf = u & 1, row = wk.r0 + r;
        const float2 *st = stats + buf * UNIT;
        int lo, hi;
        uint32_t len;
        if constexpr (MODE == MODE_K2) {
            const int i = row - kp.off2 + wk.e;
            const bool ok = row < kp.nk2 && i >= 0 && i < kp.n;
            if (wk.first()) {
                const int64_t o = ((int64_t)b * kp.hq + wk.head()) * kp.n + (ok ? i : 0);
                lse2 = ok ? kp.lse[o] * LOG2E : 0.f;
                dl = ok ? kp.delta[o] : 0.f;
            }
            const int d1 = i + kp.off1 - wk.c0;
            lo = max(0, d1 - kp.w1 + 1);
            hi = ok ? min(UNIT - 1, d1) : -1;
        } else {
            const int base = row - kp.off1 - wk.c0;            // column whose query sits at the row's key
            lo = max(max(0, base), wk.e - kp.off2 - wk.c0);
            hi = row < kp.nk1 ? min(min(UNIT - 1, base + kp.w1 - 1), wk.i_hi - wk.c0) : -1;
        }
        column_range(lo, hi, len);
        if (!warp_wait(&bars[B_S_FULL + buf], (u >> 1) & 1, abort_flag, 1)) return ERR_BWD;
        tc_fence_after();
        // sixteen columns at a time, either half from the outside in (put_terms)
#pragma unroll 2
        for (int y = 0; y < 4 / BwdCfg<MODE>::GROUPS; ++y) {
            const int half = BwdCfg<MODE>::GROUPS == 2 ? cg : y >> 1, k = half ? 3 - (y & 1) : y & 1;
            const int c0 = 16 * k;
            const uint32_t rp = lanes + 192 * buf, rg = rp + 96;
            uint32_t s[16], g[16];
            if (__all_sync(0xffffffffu, lo > c0 + 15 || (int)(lo + len) < c0)) {       // nothing valid for this warp
#pragma unroll
                for (int z = 0; z < 16; ++z) { s[z] = 0u; g[z] = 0u; }
            } else {
                tmem_ld16(rp + LOGITS + c0, s);
                tmem_ld16(rg + LOGITS + c0, g);
                tmem_wait_ld(s);
                tmem_wait_ld(g);
                const bool full = __all_sync(0xffffffffu, lo <= c0 && (int)(lo + len) >= c0 + 15);
#pragma unroll
                for (int z = 0; z < 16; ++z) {
                    const float a = __uint_as_float(s[z]) - (MODE == MODE_K2 ? lse2 : st[c0 + z].x);
                    s[z] = __float_as_uint(!full && (uint32_t)(c0 + z - lo) > len ? -CUDART_INF_F : a);
                }
#pragma unroll
                for (int z = 0; z < 16; z += 2) {
                    const float p0 = ex2(__uint_as_float(s[z])), p1 = ex2(__uint_as_float(s[z + 1]));
                    const float d0 = MODE == MODE_K2 ? dl : st[c0 + z].y, d1 = MODE == MODE_K2 ? dl : st[c0 + z + 1].y;
                    float g0, g1;
                    f2_unpack(f2_mul(f2_pack(p0, p1), f2_add(f2_pack(g[z], g[z + 1]), f2_pack(-d0, -d1))), g0, g1);
                    s[z] = __float_as_uint(p0); s[z + 1] = __float_as_uint(p1);
                    g[z] = __float_as_uint(g0); g[z + 1] = __float_as_uint(g1);
                }
            }
            put_terms(rp, k, s);
            put_terms(rg, k, g);
        }
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(&bars[B_P_FULL + buf]);
    }
    return 0;
}

// Operands and sums of one side (which = 0: A_e, K1 and U; 1: B_e, V1 and W).  Unit u of the
// operands is made when unit u - 2 is done and its product has been added up: both take the same slot.
template <int D, int MODE>
__device__ __forceinline__ int bwd_side(const BwdParams &P, int which, uint32_t tmem, uint8_t *sM, uint8_t *sN, float2 *stats, float *ring,
                                        uint64_t *bars, volatile int *abort_flag, uint32_t *most) {
    constexpr int CPR = D / 8, RPP = 128 / CPR;        // chunks of a row, rows 128 threads cover at a time
    constexpr int TASKS = UNIT / RPP;
    const KernelParams &kp = P.kp;
    const int t = threadIdx.x & 127, c = t % CPR, q0 = t / CPR;
    const int hk = blockIdx.y, b = blockIdx.z;
    const uint32_t cols = tmem + ((uint32_t)(t & 96) << 16) + 384 + 64 * which;
    const float mul = which ? 1.f : logit_factor(kp.scale, true);
    const TensorRef &tx = which ? kp.dout : kp.q, &ty = which ? kp.v2 : kp.k2, &tk = which ? kp.v1 : kp.k1;
    uint8_t *dM = sM + which * Planes<D>::bytes(ROWS), *dN = sN + which * 2 * Planes<D>::bytes(UNIT);
    uint64_t acc[D / 2], sum[MODE == MODE_K2 ? D / 2 : 1];
#pragma unroll
    for (int z = 0; z < D / 2; ++z) { acc[z] = 0; sum[MODE == MODE_K2 ? z : 0] = 0; }

    Walk<MODE> nxt(P), cur(P);
    const int row = nxt.r0 + t;                        // the row whose sums this thread keeps
    int sweeps = 0, folds = 0, err = 0;
    float most_m = 0.f, most_n = 0.f;
    float held[MODE == MODE_K1 ? TASKS : 1][8];
    if (MODE == MODE_K1 && !nxt.done()) {
#pragma unroll 1
        for (int x = 0; x < ROWS / RPP; ++x) {
            const int rr = q0 + x * RPP, j = nxt.r0 + rr;
            float k[8];
            load8(k, row_ptr(tk, b, j < kp.nk1 ? j : 0, hk) + c * 8, j < kp.nk1);
            put8<D>(dM, ROWS, rr, c, k, most_m);
        }
        fence_proxy_async_smem();
        mbar_arrive(&bars[B_M_FULL + which]);
    }
    // end of a sweep (MODE_K2): sum[] is U (W) of the thread's second key and the query e rows on
    auto fold = [&]() -> bool {
        const int e = cur.e, i = row - kp.off2 + e, h = cur.head();
        const bool ok = row < kp.nk2 && i >= 0 && i < kp.n;
        const float4 *px = reinterpret_cast<const float4 *>(row_ptr(tx, b, ok ? i : 0, h));
        const float4 *py = reinterpret_cast<const float4 *>(row_ptr(ty, b, ok ? row : 0, hk));
        const int rr = t + e - cur.e0, slot = rr & (ROWS - 1);
        const bool fresh = e == cur.ea || t == ROWS - 1, out = e == cur.eb || t == 0;
        float4 *dst = reinterpret_cast<float4 *>(ring + slot * D);
        float4 *slab = nullptr;
        if (which == 0) {
            const int es = (int)blockIdx.x % P.nsplit / P.hsplit, tile = (int)blockIdx.x / P.nsplit;
            slab = reinterpret_cast<float4 *>(P.slab + (((((size_t)b * kp.hq + h) * P.tiles + tile) * (P.nsplit / P.hsplit) + es) * (ROWS - 1 + P.epc) + rr) * D);
            // the row was another thread's in the last sweep
            if (folds > 0 && !warp_wait(&bars[B_RING], (folds - 1) & 1, abort_flag, 3)) return false;
        }
#pragma unroll
        for (int z = 0; z < D / 4; ++z) {
            const uint64_t s0 = sum[MODE == MODE_K2 ? 2 * z : 0], s1 = sum[MODE == MODE_K2 ? 2 * z + 1 : 0];
            if (ok) {
                const float4 v = __ldg(px + z);
                acc[2 * z] = f2_fma(s0, f2_pack(v.x, v.y), acc[2 * z]);
                acc[2 * z + 1] = f2_fma(s1, f2_pack(v.z, v.w), acc[2 * z + 1]);
            }
            if (which == 0) {
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f), *cell = dst + ((z ^ slot) & (D / 4 - 1));
                if (!fresh) a = *cell;
                if (ok) {
                    const float4 y = __ldg(py + z);
                    f2_unpack(f2_fma(s0, f2_pack(y.x, y.y), f2_pack(a.x, a.y)), a.x, a.y);
                    f2_unpack(f2_fma(s1, f2_pack(y.z, y.w), f2_pack(a.z, a.w)), a.z, a.w);
                }
                *(out ? slab + z : cell) = a;
            }
        }
        if (which == 0) mbar_arrive(&bars[B_RING]);
        ++folds;
#pragma unroll
        for (int z = 0; z < D / 2; ++z) sum[MODE == MODE_K2 ? z : 0] = 0;
        return true;
    };

    for (int u = 0;; ++u) {
        const bool more = !nxt.done();
        const int slot = u & 1;
        // the unit's rows, fetched before the wait (MODE_K1: the rows of q or dO once for all offsets)
        constexpr int EARLY = MODE == MODE_K2 && BwdCfg<MODE>::GROUPS == 2 ? TASKS / 2 : TASKS;
        float x[TASKS][8];
        float2 stat = make_float2(0.f, 0.f);
        auto key_row = [&](int z) {
            const int j = nxt.c0 + q0 + z * RPP;
            load8(x[z], row_ptr(tk, b, j < kp.nk1 ? j : 0, hk) + c * 8, j < kp.nk1);
        };
        if (more) {
            if constexpr (MODE == MODE_K2) {
#pragma unroll
                for (int z = 0; z < EARLY; ++z) key_row(z);
            } else {
                const int h = nxt.head();
#pragma unroll
                for (int z = 0; z < TASKS; ++z) {
                    const int i = nxt.c0 + q0 + z * RPP, k = i + kp.off2 - nxt.e;
                    if (nxt.first()) load8(held[z], row_ptr(tx, b, i <= nxt.i_hi ? i : 0, h) + c * 8, i <= nxt.i_hi);
                    const bool ok = i <= nxt.i_hi && k >= 0;
                    load8(x[z], row_ptr(ty, b, ok ? k : 0, hk) + c * 8, ok);
                }
                const int i = nxt.c0 + t;
                if (which == 0 && t < UNIT && i <= nxt.i_hi) {
                    const int64_t o = ((int64_t)b * kp.hq + h) * kp.n + i;
                    stat = make_float2(kp.lse[o] * LOG2E, kp.delta[o]);
                }
            }
        }
        if (u >= 2) {
            if (cur.done()) break;
            if (!warp_wait(&bars[B_DONE + 2 * which + slot], ((u >> 1) - 1) & 1, abort_flag, 1)) { err = ERR_BWD; break; }
            tc_fence_after();
            if constexpr (MODE == MODE_K2) add_acc<D>(cols, sum);
            else add_acc<D>(cols, acc);
            tc_fence_before();
            mbar_arrive(&bars[B_ACC_EMPTY + which]);
        }
        if (more) {
            uint8_t *d = dN + slot * Planes<D>::bytes(UNIT);
#pragma unroll
            for (int z = 0; z < TASKS; ++z) {
                if constexpr (MODE == MODE_K1) {
#pragma unroll
                    for (int w = 0; w < 8; ++w) x[z][w] = mul * held[MODE == MODE_K1 ? z : 0][w] * x[z][w];
                } else if (z == EARLY) {
#pragma unroll
                    for (int y = EARLY; y < TASKS; ++y) key_row(y);
                }
                put8<D>(d, UNIT, q0 + z * RPP, c, x[z], most_n);
            }
            if (MODE == MODE_K1 && which == 0 && t < UNIT) stats[slot * UNIT + t] = stat;
            fence_proxy_async_smem();
            mbar_arrive(&bars[B_N_FULL + 2 * which + slot]);
            if (MODE == MODE_K2 && nxt.first()) {
                const int h = nxt.head();
                if (sweeps > 0 && !warp_wait(&bars[B_M_EMPTY + which], (sweeps - 1) & 1, abort_flag, 2)) { err = ERR_BWD; break; }
                ++sweeps;
#pragma unroll 2
                for (int z = 0; z < ROWS / RPP; ++z) {
                    const int rr = q0 + z * RPP, k = nxt.r0 + rr, i = k - kp.off2 + nxt.e;
                    const bool ok = k < kp.nk2 && i >= 0 && i < kp.n;
                    float a[8], y[8];
                    load8(a, row_ptr(tx, b, ok ? i : 0, h) + c * 8, ok);
                    load8(y, row_ptr(ty, b, ok ? k : 0, hk) + c * 8, ok);
#pragma unroll
                    for (int w = 0; w < 8; ++w) a[w] = mul * a[w] * y[w];
                    put8<D>(dM, ROWS, rr, c, a, most_m);
                }
                fence_proxy_async_smem();
                mbar_arrive(&bars[B_M_FULL + which]);
            }
            nxt.next();
        }
        if (u >= 2) {
            if (MODE == MODE_K2 && cur.last() && !fold()) { err = ERR_BWD; break; }
            cur.next();
        }
    }

    put_most(&most[which], most_m);
    put_most(&most[2 + which], most_n);
    // the row's sums: final, or a partial for the reduction
    const bool bad = __any_sync(0xffffffffu, err != 0) || *abort_flag != 0;
    const int rows = MODE == MODE_K1 ? kp.nk1 : kp.nk2;
    if (row < rows) {
        const TensorRef &dst = MODE == MODE_K1 ? (which ? kp.dv1 : kp.dk1) : (which ? kp.dv2 : kp.dk2);
        // (A_e carries scale * log2(e); U does not carry the scale)
        const float fac = which ? 1.f : MODE == MODE_K1 ? logit_unfactor(kp.scale, mul) : kp.scale;
        float *part = P.part + (((((size_t)(blockIdx.x % P.nsplit) * kp.b + b) * rows + row) * kp.hk + hk) * 2 + which) * D;
        const int64_t off = elem_off(dst, b, row, hk);
#pragma unroll
        for (int z = 0; z < D / 4; ++z) {
            float v[4];
            f2_unpack(acc[2 * z], v[0], v[1]);
            f2_unpack(acc[2 * z + 1], v[2], v[3]);
#pragma unroll
            for (int w = 0; w < 4; ++w) v[w] = bad ? CUDART_NAN_F : v[w] * fac;
            if (P.nsplit > 1) store_vec<4>(part, 4 * z, false, v);
            else store_vec<4>(dst.p, off + 4 * z, kp.grad_bf16 != 0, v);
        }
    }
    // dQ rows that were given up on: those of the whole slab
    if (MODE == MODE_K2 && which == 0 && bad) {
        const int es = (int)blockIdx.x % P.nsplit / P.hsplit, tile = (int)blockIdx.x / P.nsplit, hs = (int)blockIdx.x % P.nsplit % P.hsplit;
        for (int h = hk * kp.g + kp.g * hs / P.hsplit; h < hk * kp.g + kp.g * (hs + 1) / P.hsplit; ++h) {
            float *slab = P.slab + ((((size_t)b * kp.hq + h) * P.tiles + tile) * (P.nsplit / P.hsplit) + es) * (size_t)(ROWS - 1 + P.epc) * D;
            for (int x = t; x < (ROWS - 1 + P.epc) * D; x += 128) slab[x] = CUDART_NAN_F;
        }
    }
    return err;
}

template <int D, int MODE>
__global__ void __launch_bounds__(BwdCfg<MODE>::THREADS, 1) bwd_kernel(const BwdParams P) {
    using C = BwdCfg<MODE>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = align_smem(smem_raw);
    uint8_t *sM = smem;                                           // [2]: A_e, B_e or K1, V1
    uint8_t *sN = sM + 2 * Planes<D>::bytes(ROWS);                // [2][2 slots]
    uint8_t *extra = sN + 4 * Planes<D>::bytes(UNIT);             // dQ ring, or [2 slots] lse and D of the columns
    uint64_t *bars = reinterpret_cast<uint64_t *>(extra + (MODE == MODE_K2 ? ROWS * D * 4 : 2 * UNIT * 8));
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bars + B_BAR_COUNT);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_holder + 1);
    uint32_t *most = tmem_holder + 2;            // [4] largest magnitudes of A_e and B_e (or K1 and V1), and of the operands on the other side

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    if (threadIdx.x == 0) {
        for (int x = 0; x < B_BAR_COUNT; ++x) {
            const bool one = (x >= B_M_EMPTY && x < B_M_EMPTY + 2) || (x >= B_DONE && x < B_DONE + 4);
            const bool two = x == B_S_FULL || x == B_S_FULL + 1;
            const bool compute = x == B_P_FULL || x == B_P_FULL + 1;
            mbar_init(&bars[x], one ? 1u : two ? 2u : compute ? 128u * C::GROUPS : 128u);
        }
        *abort_flag = 0;
        for (int x = 0; x < 4; ++x) most[x] = 0u;
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
    int err;
#ifdef SA2_PROF
    const long long prof_t0 = clock64();
    sa2::sm100::prof_begin();
#endif
    if (warp < 4) {
        reg_dealloc<C::REGS_ISSUE>();
        if (warp == 1 || warp == 2) err = bwd_first<D, MODE>(P, warp - 1, tmem, sM, sN, bars, abort_flag);
        else err = bwd_second<D, MODE>(P, warp == 3, tmem, sN, bars, abort_flag);
    } else if (warp < 4 + 4 * C::GROUPS) {
        if constexpr (C::REGS_COMPUTE > C::REGS_LAUNCH) reg_alloc<C::REGS_COMPUTE>();
        else reg_dealloc<C::REGS_COMPUTE>();
        err = bwd_compute<D, MODE>(P, (warp >> 2) - 1, tmem, reinterpret_cast<const float2 *>(extra), bars, abort_flag);
    } else {
        reg_alloc<C::REGS_SUM>();
        err = bwd_side<D, MODE>(P, warp >= 8 + 4 * C::GROUPS, tmem, sM, sN, reinterpret_cast<float2 *>(extra), reinterpret_cast<float *>(extra), bars, abort_flag,
                                most);
    }
    if (err) atomicOr(P.status, err);
    SA2_PROF_ADD(0, clock64() - prof_t0);
    SA2_PROF_END();
    tc_fence_before();
    __syncthreads();
    // (dP is the product of most[1] and most[3], G is of its size)
    if (threadIdx.x < 5 && out_of_range(threadIdx.x < 4 ? __uint_as_float(most[threadIdx.x]) : fminf(1.f, __uint_as_float(most[1])) * __uint_as_float(most[3])))
        P.redo[blockIdx.z] = 1;
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

// ---------------------------------------------------------------------------
// Sums of the partials, one thread per 4 channels of a row:
//   dq[i]        = scale * sum over the offset ranges and the tiles whose slab holds row i
//   dk2, dv2[k]  = sum over the splits (more than one), dk1, dv1[j] likewise
// ---------------------------------------------------------------------------
struct ReduceParams {
    KernelParams kp;
    const float *slab, *part_k2, *part_k1;
    int tiles, esplit, epc;       // of MODE_K2
    int k2_splits, k1_splits;     // 0: nothing to add up
    int dq;                       // dQ is asked for
};
// G threads take the offset ranges or splits of a piece by turns, and their sums are added in order: where splits are many, the rows
// are few (b1 n128 h2 d32 full causal, 64 ranges: 26 -> 6 us with eight).
template <int D, int G>
__global__ void __launch_bounds__(256) reduce_kernel(const ReduceParams R) {
    const KernelParams &kp = R.kp;
    constexpr int TPR = D / 4, RPB = 256 / (TPR * G);        // threads of a row, rows of a block
    __shared__ float4 sums[G > 1 ? 2 : 1][G > 1 ? 256 : 1];
    const int c = (int)(threadIdx.x % TPR) * 4, g = (int)threadIdx.x / TPR % G;
    int64_t idx = (int64_t)blockIdx.x * RPB + threadIdx.x / (TPR * G);
    const bool gbf16 = kp.grad_bf16 != 0;
    const int64_t nq = R.dq ? (int64_t)kp.b * kp.n * kp.hq : 0;
    const int64_t n2 = R.k2_splits ? (int64_t)kp.b * kp.nk2 * kp.hk : 0, n1 = R.k1_splits ? (int64_t)kp.b * kp.nk1 * kp.hk : 0;
    float v[2][4] = {};
    auto add = [](float (&a)[4], const float4 &x) { a[0] += x.x; a[1] += x.y; a[2] += x.z; a[3] += x.w; };
    // the first of the G threads of a piece has the sum
    auto gather = [&](int y) {
        if constexpr (G > 1) {
            sums[y][threadIdx.x] = make_float4(v[y][0], v[y][1], v[y][2], v[y][3]);
            __syncthreads();
            if (g == 0)
                for (int x = 1; x < G; ++x) add(v[y], sums[y][threadIdx.x + x * TPR]);
        }
    };
    const bool is_q = idx < nq, is_2 = !is_q && idx < nq + n2, is_1 = !is_q && !is_2 && idx < nq + n2 + n1;
    if (is_q) {
        const int h = (int)(idx % kp.hq), i = (int)(idx / kp.hq % kp.n), b = (int)(idx / ((int64_t)kp.hq * kp.n));
        const int rows = ROWS - 1 + R.epc;
        const float *slab = R.slab + ((size_t)b * kp.hq + h) * R.tiles * R.esplit * rows * D + c;
        // (unrolled for the loads in flight; the order of the sum is that of the loop)
#pragma unroll 4
        for (int es = g; es < R.esplit; es += G) {
            const int e0 = es * R.epc, e1 = min(kp.w2, e0 + R.epc);
            // second keys i + off2 - e of the range, from the last tile that holds one to the first
            const int k_hi = i + kp.off2 - e0, k_lo = max(0, i + kp.off2 - e1 + 1), last = k_hi < 0 ? -1 : k_hi / ROWS, first = k_lo / ROWS;
            auto row = [&](int tile) {
                return *reinterpret_cast<const float4 *>(slab + (((size_t)tile * R.esplit + es) * rows + k_hi - tile * ROWS) * D);
            };
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
            if (last >= first) x = row(last);
            if (last > first) y = row(last - 1);
            add(v[0], x);
            add(v[0], y);
            for (int tile = last - 2; tile >= first; --tile) add(v[0], row(tile));
        }
    } else if (is_2 || is_1) {
        idx -= is_2 ? nq : nq + n2;
        const int64_t all = is_2 ? n2 : n1;
        const int splits = is_2 ? R.k2_splits : R.k1_splits;
        const float *part = is_2 ? R.part_k2 : R.part_k1;
#pragma unroll 4
        for (int s = g; s < splits; s += G) {
            const float *src = part + ((s * all + idx) * 2) * D + c;
            add(v[0], *reinterpret_cast<const float4 *>(src));
            add(v[1], *reinterpret_cast<const float4 *>(src + D));
        }
    }
    gather(0);
    gather(1);
    if (g != 0 || !(is_q || is_2 || is_1)) return;
    if (is_q) {
        const int h = (int)(idx % kp.hq), i = (int)(idx / kp.hq % kp.n), b = (int)(idx / ((int64_t)kp.hq * kp.n));
#pragma unroll
        for (int z = 0; z < 4; ++z) v[0][z] *= kp.scale;
        store_vec<4>(kp.dq.p, elem_off(kp.dq, b, i, h) + c, gbf16, v[0]);
        return;
    }
    const int rows = is_2 ? kp.nk2 : kp.nk1;
    const int hk = (int)(idx % kp.hk), row = (int)(idx / kp.hk % rows), b = (int)(idx / ((int64_t)kp.hk * rows));
    const TensorRef &dk = is_2 ? kp.dk2 : kp.dk1, &dv = is_2 ? kp.dv2 : kp.dv1;
    store_vec<4>(dk.p, elem_off(dk, b, row, hk) + c, gbf16, v[0]);
    store_vec<4>(dv.p, elem_off(dv, b, row, hk) + c, gbf16, v[1]);
}

}  // namespace f32
}  // namespace sa2
