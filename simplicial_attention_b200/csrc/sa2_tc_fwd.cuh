// Forward kernel on the 5th-generation tensor cores (tcgen05 + TMEM + TMA),
// bf16 operands, fp32 accumulation, head dims 32 and 64.
//
// A tile is 128 (query row, second-key offset) pairs of one (batch, query head): RI query rows times
// RE = 128 / RI offsets e = i - k, row r = s * RI + (i - i0) holding e = RE * t + s in "sweep" t.  Per sweep
// the kernel forms A[r,:] = q_i * k2_{i-e} (bf16, in shared memory), multiplies it against the
// TMA-staged K1 window of the RI rows (S = A K1^T, 64 keys a unit), turns S into P = exp2(c*S - ref) in
// registers, writes P to TMEM as bf16 and feeds it as the A operand of W += P V1 (V1 unit as an MN-major B
// operand).  At the end of a sweep the row owner adds v2_{i-e} * W to its output registers; at the end of
// the tile the RE partial outputs of a query row are merged through shared memory.  The softmax is joint
// over all (j, e).
//
// Why pairs: the window of RI rows is w1 + RI - 1 keys, so a small RI wastes fewer masked columns (w1 = 512:
// 576 columns at RI = 64, 640 at RI = 128), a short sequence is spread over more CTAs of fewer sweeps each,
// and a single new token (generation) takes 16 offsets of its window at a time: 16 live rows of a tile of RI = 8, the
// smallest.  fwd_ri_log2() picks RI.
//
// Warp roles (512 threads, four aligned warpgroups):
//   warp 0, 1     issue the tcgen05.mma stream of group 0 / group 1 (warp 1 owns the TMEM allocation)
//   warp 2, 3     TMA producers: second keys of the tile and K1 units, second values and V1
//                 units (units are resident if the window fits, else a ring walked once per pair of sweeps)
//   warps 4-7     output group, one thread per row: builds the A row of each group's next sweep as soon as the
//                 last S product of its current sweep has completed, and folds v2 * W of the finished sweep
//   warps 8-11    softmax group 0: even sweeps, one thread per row
//   warps 12-15   softmax group 1: odd sweeps, one thread per row
// An even and an odd sweep are in flight together, so while one group runs the exponentials of its unit the
// tensor cores work for the other and each SM sub-partition has two softmax warps to hide latencies.
//
// A unit is 64 keys.  TMEM columns of group g, from 256 g: S 2 x 64, P (bf16) 2 x 32, W 64.
//
// Bound: the two softmax groups, busy ~85 % of a unit's ~900 cycles (two warps a scheduler, 512 MUFU cycles a unit) and
// mostly in phase with each other on the MUFU pipe.  A softmax warp has one barrier wait and one arrival per unit -
// the issuing thread of a group alternates P V1 of unit u and S of unit u + 2, whose completion therefore also says
// that the P columns are free - and which 32-column chunks need no mask, or are seen by nobody, is decided from
// warp-uniform bounds without votes.
// Measured: b4 n4096 h8 d64 w512/32 1.26 -> 0.95 ms (543 TFLOP/s), b2 n1024 0.179 -> 0.139 ms; one new row of b1 h8 behind a
// full window 0.19 -> 0.017 ms.
// Measured and not kept, where this form takes 0.96 (or, earlier, 1.12) ms: A in TMEM with one P buffer (1.5 against 1.12),
// 128-key units (1.4), S and P V1 from separate issuing threads (1.15), S(u + 2) before P V1(u) (1.19), ordering the
// softmax groups against each other (1.04 against 0.96), A and W double-buffered (0.98), an output group that takes its
// events as they come (1.01).
//
// SPLIT (head dim 32, and head dim 64 with w1 > 513: see fwd_split): A and P are each a bf16 value and a bf16 rest, so S and
// P V1 take two products per K step instead of one, with the rests of P over the S columns they come from.  The softmax
// groups pack twice as many words, which is what the time goes to: b1 n3001 h8 d64 w1024/16 0.207 -> 0.250 ms, b4 n4096 h8 d32
// w512/32 0.90 -> 1.08 ms against rounded operands; 4.15 and 12.6 ms on the fp32 kernels.
//
// Reference handling: probabilities are computed against a per-row reference
// that only moves when it must, so the W accumulator in TMEM normally never
// needs a rescale; bf16 has fp32's exponent range, so P may exceed 1 by many
// orders of magnitude without loss.  When the probabilities of a unit sum to
// more than 2^64 (always true for a row's very first unit, whose reference is
// -inf) the warp takes a slow path: exact unit maximum, rescale of the row's
// partial sums (including W in TMEM), recomputation of P.
#pragma once
#include "sa2_tc_common.cuh"

namespace sa2 {
namespace tc {

constexpr int FWD_THREADS = 512;
// Register hand-over between warpgroups (launch: 128 per thread; the budgets must add up to at most 4 * 128, or
// the growing group never returns from its setmaxnreg).
constexpr int FWD_REGS_LAUNCH = 128, FWD_REGS_ISSUE = 56, FWD_REGS_SOFTMAX = 120, FWD_REGS_OUT = 216;
static_assert(FWD_REGS_ISSUE + 2 * FWD_REGS_SOFTMAX + FWD_REGS_OUT <= 4 * FWD_REGS_LAUNCH, "register pool must balance");
static_assert(FWD_REGS_SOFTMAX < FWD_REGS_LAUNCH, "the softmax groups release registers");
constexpr int FWD_UNIT = 64;                                  // first-key rows of a unit
constexpr uint32_t FWD_UNIT_BYTES = FWD_UNIT * 128;           // its K1 (or V1) rows, 128 bytes each
constexpr int FWD_MAX_SLOTS = 12;
constexpr int FWD_WIN_ROWS = 128;                             // most second-key rows staged in shared memory

enum FwdBar {
    BAR_KV_FULL = 0,                              // [FWD_MAX_SLOTS] K1 and V1 rows of the unit have landed
    BAR_KV_FREE = BAR_KV_FULL + FWD_MAX_SLOTS,    // [FWD_MAX_SLOTS] both groups' products on the unit are done
    BAR_WIN_FULL = BAR_KV_FREE + FWD_MAX_SLOTS,   // second-key and second-value rows have landed
    BAR_A_FULL = BAR_WIN_FULL + 1,                // [2] per group
    BAR_A_FREE = BAR_A_FULL + 2,                  // [2] every S product of the sweep has completed
    BAR_S_FULL = BAR_A_FREE + 2,                  // [4] group * 2 + buffer
    BAR_P_FULL = BAR_S_FULL + 4,                  // [4] P of the unit is in TMEM and its S has been read (one per
                                                  // buffer: a warp may be a unit ahead of another)
    BAR_PV_DONE = BAR_P_FULL + 4,                 // [2] W += P V1 of the unit has completed
    BAR_W_FULL = BAR_PV_DONE + 2,                 // [2]
    BAR_W_EMPTY = BAR_W_FULL + 2,                 // [2]
    BAR_REF_FULL = BAR_W_EMPTY + 2,               // [2] the sweep's final reference is in shared memory
    BAR_COUNT = BAR_REF_FULL + 2
};

struct FwdParams {
    KernelParams kp;
    int ri_log2;     // query rows per tile
    int nslots;      // K1/V1 units in shared memory
    int win_boxes;   // 32-row boxes of staged k2 (and v2) rows; 0: read from global memory
    float c;         // scale * log2(e)
    int *status;     // device status word
};

// at least 120 KB: one CTA per SM, so the 512-column TMEM allocation never waits for a co-resident CTA; at least
// three slots: the merge of the row partials (128 rows of D + 4 floats) reuses them
inline size_t fwd_smem_bytes(int nslots, int win_boxes, int a_tiles) {
    const size_t need = 1024 + (size_t)(nslots > 3 ? nslots : 3) * 2 * FWD_UNIT_BYTES + (size_t)win_boxes * 2 * 4096 + a_tiles * TILE_BYTES +
                        FWD_STATS_FLOATS * 4 + BAR_COUNT * 8 + 64;
    return need > 120 * 1024 ? need : 120 * 1024;
}

// The A rows of a group: one tile, of which head dim 32 uses half a row for the rounded products and, with SPLIT, the other
// half for what the rounding left; head dim 64 puts that into a second tile.
template <int D, bool SPLIT> struct FwdA {
    static constexpr int TILES = SPLIT && D == 64 ? 2 : 1;             // per group
    static constexpr uint32_t BYTES = TILES * TILE_BYTES;
    static constexpr uint32_t REST = D == 64 ? TILE_BYTES : 64;        // bytes from an element to its rest
};

struct FwdGeom {
    int i0, i_last, ri, ri_log2, re;
    int jbase;        // unit x of a sweep covers rows jbase + 64 x ... + 63
    int upe;          // units per sweep
    int nsw[2];       // sweeps of each group
    int win0;         // position of the first staged second-key row
    bool resident;    // every unit of the window has its own slot
};

template <class PT>
__device__ __forceinline__ FwdGeom fwd_geom(const PT &P) {
    FwdGeom g;
    const KernelParams &kp = P.kp;
    g.ri_log2 = P.ri_log2;
    g.ri = 1 << P.ri_log2;
    g.re = TQ >> P.ri_log2;
    g.i0 = blockIdx.x << P.ri_log2;
    g.i_last = min(g.i0 + g.ri - 1, kp.n - 1);
    const int jend = g.i_last + kp.off1 + 1, jlow = max(0, g.i0 + kp.off1 - kp.w1 + 1);
    g.upe = (jend - jlow + FWD_UNIT - 1) / FWD_UNIT;
    g.jbase = jend - FWD_UNIT * g.upe;                 // may be negative: TMA reads zeros there
    const int ne = min(kp.w2, g.i_last + kp.off2 + 1);
    const int nsweeps = (ne + g.re - 1) >> (7 - P.ri_log2);
    g.nsw[0] = (nsweeps + 1) / 2;
    g.nsw[1] = nsweeps / 2;
    g.win0 = g.i0 + kp.off2 - (kp.w2 - 1);
    g.resident = g.upe <= P.nslots;
    return g;
}

// Where the units of a walk live: in a resident window unit w has slot w and is loaded once; a ring gives the x-th
// unit of the walk (x counts units over pairs of sweeps) slot x % nslots.
struct FwdSlot {
    int slot = 0, use = 0;       // `use`: how often the slot has been used before (ring)
    __device__ __forceinline__ void next(const FwdParams &P, const FwdGeom &g, int w) {
        if (g.resident) slot = w + 1 == g.upe ? 0 : w + 1;
        else if (++slot == P.nslots) { slot = 0; ++use; }
    }
};

// ------------------------------------------------------------------ TMA producers (warps 2 and 3)
__device__ __forceinline__ int fwd_producer(const FwdParams &P, const FwdGeom &g, const CUtensorMap *map, const CUtensorMap *map2,
                                            uint8_t *dst, uint8_t *win, uint64_t *bars, volatile int *abort_flag) {
    const int b = blockIdx.z, hk = blockIdx.y / P.kp.g;
    const int items = g.resident ? g.upe : g.nsw[0] * g.upe;
    FwdSlot s;
    int w = 0;
    auto load = [&]() -> bool {
        if (s.use >= 1 && !mbar_wait_warp(&bars[BAR_KV_FREE + s.slot], (s.use - 1) & 1, abort_flag, 32, 1)) return false;
        if (elect_one()) {
            mbar_arrive_expect_tx(&bars[BAR_KV_FULL + s.slot], FWD_UNIT_BYTES);
            tma_load_4d(dst + s.slot * FWD_UNIT_BYTES, map, &bars[BAR_KV_FULL + s.slot], 0, hk, g.jbase + FWD_UNIT * w, b);
        }
        s.next(P, g, w);
        if (++w == g.upe) w = 0;
        return true;
    };
    if (P.win_boxes > 0 && elect_one()) {
        mbar_arrive_expect_tx(&bars[BAR_WIN_FULL], P.win_boxes * 4096);
        for (int bx = 0; bx < P.win_boxes; ++bx) tma_load_4d(win + bx * 4096, map2, &bars[BAR_WIN_FULL], 0, hk, g.win0 + 32 * bx, b);
    }
    for (int x = 0; x < items; ++x)
        if (!load()) return ERR_FWD_PRODUCER;
    // every load must have landed before the CTA may exit, even if the consumers gave up
    if (P.win_boxes > 0 && !mbar_wait_warp(&bars[BAR_WIN_FULL], 0, abort_flag, 32)) return ERR_FWD_PRODUCER;
    for (int x = max(0, items - P.nslots); x < items; ++x)
        if (!mbar_wait_warp(&bars[BAR_KV_FULL + x % P.nslots], (x / P.nslots) & 1, abort_flag, 32)) return ERR_FWD_PRODUCER;
    return 0;
}

// ------------------------------------------------------------------ MMA issuers (warps 0 and 1)
// Warp g issues for group g: the two groups touch disjoint TMEM columns and only read shared memory,
// so their MMA streams need no ordering between them.  P V1 of unit u goes before S of unit u + 2, whose
// completion therefore covers it (and the sweep after the next needs its A rows by then, whose builder waits for
// the W that P V1 completes).
template <int D, bool SPLIT>
__device__ __forceinline__ int fwd_mma(const FwdParams &P, const FwdGeom &g, int grp, uint32_t tmem, uint8_t *sK, uint8_t *sV, uint8_t *sA,
                                       uint64_t *bars, volatile int *abort_flag) {
    constexpr uint32_t IDESC_S = idesc_bf16(128, FWD_UNIT, false, false);
    constexpr uint32_t IDESC_PV = idesc_bf16(128, 64, false, true);    // (head dim 32: the upper 32 channels are zeros)
    const uint64_t dK = smem_desc_sw128(smem_u32(sK)), dV = smem_desc_sw128(smem_u32(sV));
    const uint64_t dA = smem_desc_sw128(smem_u32(sA) + grp * FwdA<D, SPLIT>::BYTES);
    const uint32_t tS = tmem + grp * 256, tP = tS + 128, tW = tS + 192;
    const int upe = g.upe, n = g.nsw[grp] * upe;
    FwdSlot ss, ps;
    int s_k = 0, s_w = 0, p_k = 0, p_w = 0;             // sweep and unit of the next S and of the next P V1

    auto issue_s = [&](int u) -> bool {
        if (s_w == 0 && !mbar_wait_warp(&bars[BAR_A_FULL + grp], s_k & 1, abort_flag, 0, 1)) return false;
        if ((s_k == 0 || !g.resident) && !mbar_wait_warp(&bars[BAR_KV_FULL + ss.slot], ss.use & 1, abort_flag, 0, 4)) return false;
        tc_fence_after();
        const uint64_t kt = dK + (uint64_t)((ss.slot * FWD_UNIT_BYTES) >> 4);
        const uint32_t d = tS + (u & 1) * 64;
        if (elect_one()) {
#pragma unroll
            for (int st = 0; st < D / 16; ++st) mma_ss(d, dA + st * 2, kt + st * 2, IDESC_S, st > 0 ? 1u : 0u);
            if constexpr (SPLIT) {
#pragma unroll
                for (int st = 0; st < D / 16; ++st) mma_ss(d, dA + (FwdA<D, SPLIT>::REST >> 4) + st * 2, kt + st * 2, IDESC_S, 1u);
            }
            tc_commit(&bars[BAR_S_FULL + grp * 2 + (u & 1)]);
            if (s_w == upe - 1) tc_commit(&bars[BAR_A_FREE + grp]);      // the A rows may be rebuilt
        }
        ss.next(P, g, s_w);
        if (++s_w == upe) { s_w = 0; ++s_k; }
        return true;
    };
    for (int u = 0; u < 2 && u < n; ++u)
        if (!issue_s(u)) return ERR_FWD_MMA;
    for (int u = 0; u < n; ++u) {
        if (p_w == 0 && p_k >= 1 && !mbar_wait_warp(&bars[BAR_W_EMPTY + grp], (p_k - 1) & 1, abort_flag, 0, 3)) return ERR_FWD_MMA;
        if (!mbar_wait_warp(&bars[BAR_P_FULL + grp * 2 + (u & 1)], (u >> 1) & 1, abort_flag, 0, 2)) return ERR_FWD_MMA;
        tc_fence_after();
        const uint64_t vt = dV + (uint64_t)((ps.slot * FWD_UNIT_BYTES) >> 4);
        const uint32_t a = tP + (u & 1) * 32;
        if (elect_one()) {
#pragma unroll
            for (int st = 0; st < 4; ++st) mma_ts(tW, a + st * 8, vt + st * 128, IDESC_PV, (p_w > 0 || st > 0) ? 1u : 0u);
            if constexpr (SPLIT) {          // the rests of P lie over the S they come from
#pragma unroll
                for (int st = 0; st < 4; ++st) mma_ts(tW, tS + (u & 1) * 64 + st * 8, vt + st * 128, IDESC_PV, 1u);
            }
            tc_commit(&bars[BAR_PV_DONE + grp]);
            if (!g.resident) tc_commit(&bars[BAR_KV_FREE + ps.slot]);
            if (p_w == upe - 1) tc_commit(&bars[BAR_W_FULL + grp]);
        }
        ps.next(P, g, p_w);
        if (++p_w == upe) { p_w = 0; ++p_k; }
        if (u + 2 < n) {
            // S of unit u + 2 goes where the rests of P of unit u are; the softmax group has unit u + 1 to work on meanwhile
            if (SPLIT && !mbar_wait_warp(&bars[BAR_PV_DONE + grp], u & 1, abort_flag, 0, 5)) return ERR_FWD_MMA;
            if (!issue_s(u + 2)) return ERR_FWD_MMA;
        }
    }
    // The ring follows group 0's walk.  With an odd number of sweeps group 1 has one sweep less: it lets the
    // units of that last sweep pass, so that every slot still collects two releases.
    if (!g.resident) {
        for (int x = n; x < g.nsw[0] * upe; ++x, ps.next(P, g, 0)) {
            if (!mbar_wait_warp(&bars[BAR_KV_FULL + ps.slot], ps.use & 1, abort_flag, 32)) return ERR_FWD_MMA;
            if (elect_one()) mbar_arrive(&bars[BAR_KV_FREE + ps.slot]);
        }
    }
    return 0;
}

// ------------------------------------------------------------------ softmax groups (warps 8-11, 12-15)
// Which rows the 32 rows of a warp are, in terms that are the same for all its lanes.
struct FwdWarpRows {
    int imin, imax;     // query rows (imax may lie past the end of the sequence)
    int emin, emax;     // offsets of the rows in sweep 0
    int some0, some1;   // 32-key chunks (counted from jbase) that some row sees: some0 <= x <= some1
    int full0, full1;   // chunks that every row sees whole
};
__device__ __forceinline__ FwdWarpRows fwd_warp_rows(const KernelParams &kp, const FwdGeom &g) {
    const int first = __shfl_sync(0xffffffffu, ((int)threadIdx.x >> 5) & 3, 0) * 32;      // warp-uniform
    FwdWarpRows w;
    const int span = min(32, g.ri);
    w.imin = g.i0 + (first & (g.ri - 1));
    w.imax = w.imin + span - 1;
    w.emin = first >> g.ri_log2;
    w.emax = (first + 31) >> g.ri_log2;
    const int jlo = max(0, w.imin + kp.off1 - kp.w1 + 1), jlo_all = max(0, w.imax + kp.off1 - kp.w1 + 1);    // any / every row from
    w.some0 = max(0, jlo - g.jbase) >> 5;
    w.some1 = (w.imax + kp.off1 - g.jbase) >> 5;
    w.full0 = (max(0, jlo_all - g.jbase) + 31) >> 5;
    w.full1 = ((w.imin + kp.off1 - g.jbase + 1) >> 5) - 1;
    return w;
}

// where the rests of a chunk go: their own words, or (never written) the rounded ones
template <bool SPLIT, int N> __device__ __forceinline__ uint32_t (&fwd_rest(uint32_t (&rest)[N], uint32_t (&pk)[16]))[16] {
    if constexpr (SPLIT) return rest;
    else return pk;
}

template <bool SPLIT>
__device__ __forceinline__ int fwd_softmax(const FwdParams &P, const FwdGeom &g, int grp, uint32_t tmem, int d_w, float *stats,
                                           uint64_t *bars, volatile int *abort_flag) {
    const KernelParams &kp = P.kp;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = (warp & 3) * 32 + lane;            // row of the tile = TMEM lane
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + grp * 256;
    const int i = g.i0 + (r & (g.ri - 1)), e0 = r >> g.ri_log2;
    const FwdWarpRows wr = fwd_warp_rows(kp, g);
    const float c = P.c;
    const int upe = g.upe, nsw = g.nsw[grp];
    float *ref_slot = stats + grp * 256 + r;          // + 128 * (sweep parity)

    const uint32_t w_addr = lane_addr + 192;

    float ref = -CUDART_INF_F, l = 0.f;
    int u = 0;
    for (int k = 0; k < nsw; ++k) {
        const int eb = g.re * (2 * k + grp);
        // every row of the warp pairs with a second key in this sweep / no row does
        const bool all_ok = wr.imax < kp.n && eb + wr.emax < kp.w2 && wr.imin + kp.off2 - eb - wr.emax >= 0;
        const bool none_ok = wr.imin >= kp.n || eb + wr.emin >= kp.w2 || wr.imax + kp.off2 - eb - wr.emin < 0;
        const bool row_ok = i < kp.n && eb + e0 < kp.w2 && i + kp.off2 - eb - e0 >= 0;
        const int full0 = all_ok ? wr.full0 : 1 << 30, some1 = none_ok ? -1 : wr.some1;
#pragma unroll 1
        for (int w = 0; w < upe; ++w, ++u) {
            const int j0 = g.jbase + FWD_UNIT * w, buf = u & 1;
            const uint32_t s_addr = lane_addr + buf * 64, p_addr = lane_addr + 128 + buf * 32;
            if (!warp_wait(&bars[BAR_S_FULL + grp * 2 + buf], (u >> 1) & 1, abort_flag, 1)) return ERR_FWD_SOFTMAX;
            tc_fence_after();
            // valid columns of this row: lo < col <= hi
            const int d1 = i + kp.off1 - j0, hi = row_ok ? d1 : -1, lo = max(d1 - kp.w1, -j0 - 1);
            float sum = 0.f;
            uint32_t rest[2][SPLIT ? 16 : 1];         // SPLIT: held until S need not be read again
#pragma unroll
            for (int ch = 0; ch < 2; ++ch) {
                uint32_t s[32], pk[16];
                uint32_t (&pr)[16] = fwd_rest<SPLIT>(rest[ch], pk);
                tmem_ld32(s_addr + ch * 32, s);
                const int x = 2 * w + ch;            // 32-key chunk of the window
                tmem_wait_ld(s);
                if (x >= full0 && x <= wr.full1) {
                    sum += fwd_probs32<SPLIT>(s, pk, pr, c, ref, true, 0, 0, 0);
                } else if (x >= wr.some0 && x <= some1) {
                    sum += fwd_probs32<SPLIT>(s, pk, pr, c, ref, false, ch * 32, lo, hi);
                } else {
#pragma unroll
                    for (int z = 0; z < 16; ++z) { pk[z] = 0u; pr[z] = 0u; }
                }
                tmem_st16(p_addr + ch * 16, pk);
            }
            const bool exceed = !(sum <= 1.8446744e19f);       // above 2^64, inf or NaN
            if (__any_sync(0xffffffffu, exceed)) {
                // ---- slow path (whole warp): exact maximum of this unit, rescale, recompute
                float mx = -CUDART_INF_F;
#pragma unroll 1
                for (int ch = 0; ch < 2; ++ch) {
                    uint32_t s[32];
                    tmem_ld32(s_addr + ch * 32, s);
                    tmem_wait_ld(s);
#pragma unroll
                    for (int x = 0; x < 32; ++x) {
                        const int col = ch * 32 + x;
                        if (col > lo && col <= hi) mx = fmaxf(mx, __uint_as_float(s[x]) * c);
                    }
                }
                float f = 1.f;
                if (exceed) {
                    const float nref = fmaxf(mx, LOWEST_REF);
                    f = ex2(ref - nref);                       // 0 when ref was -inf
                    l *= f;
                    ref = nref;     // the output thread rescales its accumulator when it sees the new reference
                }
                if (w > 0) {
                    // W of this sweep already holds partial sums against the old reference
                    if (!warp_wait(&bars[BAR_PV_DONE + grp], (u - 1) & 1, abort_flag)) return ERR_FWD_SOFTMAX;
                    tc_fence_after();
#pragma unroll 1
                    for (int ch = 0; ch < d_w; ch += 32) {
                        uint32_t wv[32];
                        tmem_ld32(w_addr + ch, wv);
                        tmem_wait_ld(wv);
#pragma unroll
                        for (int x = 0; x < 32; ++x) wv[x] = __float_as_uint(__uint_as_float(wv[x]) * f);
                        tmem_st32(w_addr + ch, wv);
                    }
                }
                tmem_wait_st();
                sum = 0.f;
#pragma unroll (SPLIT ? 2 : 1)
                for (int ch = 0; ch < 2; ++ch) {
                    uint32_t s[32], pk[16];
                    uint32_t (&pr)[16] = fwd_rest<SPLIT>(rest[ch], pk);
                    tmem_ld32(s_addr + ch * 32, s);
                    tmem_wait_ld(s);
                    sum += fwd_probs32<SPLIT>(s, pk, pr, c, ref, false, ch * 32, lo, hi);
                    tmem_st16(p_addr + ch * 16, pk);
                }
            }
            if constexpr (SPLIT) {
                tmem_st16(s_addr, rest[0]);
                tmem_st16(s_addr + 16, rest[1]);
            }
            l += sum;
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(&bars[BAR_P_FULL + grp * 2 + buf]);
        }
        // W of the sweep is expressed against the reference the row has now.  The output thread has read the
        // slot of sweep k - 2 before it released that sweep's W; waiting for the release of sweep
        // k - 1 also keeps this barrier from running two phases ahead of its reader.
        if (k >= 1 && !warp_wait(&bars[BAR_W_EMPTY + grp], (k - 1) & 1, abort_flag, 3)) return ERR_FWD_SOFTMAX;
        ref_slot[(k & 1) * 128] = ref;
        mbar_arrive(&bars[BAR_REF_FULL + grp]);
    }
    stats[512 + grp * 128 + r] = l;
    stats[768 + grp * 128 + r] = ref;
    return 0;
}

// ------------------------------------------------------------------ output group (warps 4-7)
// Thread r owns row r of the tile: it builds the row of every A and accumulates the row's output against the
// larger of the references the two groups have reported (`ref_o`).
template <int D, bool SPLIT>
__device__ __forceinline__ int fwd_output(const FwdParams &P, const FwdGeom &g, uint32_t tmem, uint64_t (&o)[D / 2], float &ref_o,
                                          const uint8_t *sWin, uint8_t *sA, const float *stats, uint64_t *bars, volatile int *abort_flag) {
    constexpr int NC = D / 8;                          // 16-byte chunks of a row
    const KernelParams &kp = P.kp;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = (warp & 3) * 32 + lane;
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int h = blockIdx.y, b = blockIdx.z, hk = h / kp.g;
    const int i = g.i0 + (r & (g.ri - 1)), e0 = r >> g.ri_log2;
    const bool row_ok = i < kp.n;
    const __nv_bfloat16 *k2 = reinterpret_cast<const __nv_bfloat16 *>(kp.k2.p);
    const __nv_bfloat16 *v2 = reinterpret_cast<const __nv_bfloat16 *>(kp.v2.p);
    const bool staged = P.win_boxes > 0;
    const uint8_t *sWinV = sWin + P.win_boxes * 4096;

    uint4 qv[NC];
    const __nv_bfloat16 *qrow = reinterpret_cast<const __nv_bfloat16 *>(kp.q.p) + elem_off(kp.q, b, row_ok ? i : 0, h);
#pragma unroll
    for (int cc = 0; cc < NC; ++cc) qv[cc] = row_ok ? __ldg(reinterpret_cast<const uint4 *>(qrow + cc * 8)) : make_uint4(0u, 0u, 0u, 0u);

    // this thread's row of A = q_i * k2_{i-e} for the group's sweep k; the products are formed before the wait for
    // the stage (`bar`, unless null)
    auto build_a = [&](int grp, int k, uint64_t *bar, uint32_t parity) -> bool {
        const int e = g.re * (2 * k + grp) + e0, kk = i + kp.off2 - e;
        const bool ok = row_ok && e < kp.w2 && kk >= 0;
        const int wr = kk - g.win0;
        const __nv_bfloat16 *krow = k2 + elem_off(kp.k2, b, ok ? kk : 0, hk);
        uint8_t *dst = sA + (size_t)grp * FwdA<D, SPLIT>::BYTES;
        uint4 a[NC], rest[SPLIT ? NC : 1];
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
            uint4 kv = make_uint4(0u, 0u, 0u, 0u);
            if (ok) kv = staged ? *reinterpret_cast<const uint4 *>(sWin + sw128_offset(wr, cc)) : __ldg(reinterpret_cast<const uint4 *>(krow + cc * 8));
            a[cc].x = mul_bf16x2(qv[cc].x, kv.x); a[cc].y = mul_bf16x2(qv[cc].y, kv.y);
            a[cc].z = mul_bf16x2(qv[cc].z, kv.z); a[cc].w = mul_bf16x2(qv[cc].w, kv.w);
            if constexpr (SPLIT) rest[cc] = mul_rest_bf16x8(qv[cc], kv, a[cc]);
        }
        if (bar && !warp_wait(bar, parity, abort_flag, 1)) return false;
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) *reinterpret_cast<uint4 *>(dst + sw128_offset(r, cc)) = a[cc];
        if constexpr (SPLIT) {
#pragma unroll
            for (int cc = 0; cc < NC; ++cc)
                *reinterpret_cast<uint4 *>(dst + (D == 64 ? TILE_BYTES : 0) + sw128_offset(r, cc + (D == 64 ? 0 : 4))) = rest[cc];
        }
        fence_proxy_async_smem();
        mbar_arrive(&bars[BAR_A_FULL + grp]);
        return true;
    };

    // o += v2_{i-e} * W (TMEM), with o held against the larger reference seen so far
    auto drain = [&](int grp, int k) -> bool {
        const int e = g.re * (2 * k + grp) + e0, kk = i + kp.off2 - e;
        const bool row = row_ok && e < kp.w2 && kk >= 0;
        const int wr = kk - g.win0;
        const __nv_bfloat16 *vrow = v2 + elem_off(kp.v2, b, row ? kk : 0, hk);
        if (!warp_wait(&bars[BAR_REF_FULL + grp], k & 1, abort_flag, 2)) return false;
        const float ref_w = stats[grp * 256 + (k & 1) * 128 + r];
        if (!warp_wait(&bars[BAR_W_FULL + grp], k & 1, abort_flag, 3)) return false;
        tc_fence_after();
        const bool ok = row && ref_w > -CUDART_INF_F;
        float fw = 1.f;
        if (ok) {
            if (ref_w > ref_o) {
                const float f = ex2(ref_o - ref_w);              // 0 while the accumulator is still empty
                const uint64_t f2 = f2_pack(f, f);
#pragma unroll
                for (int x = 0; x < D / 2; ++x) o[x] = f2_mul(o[x], f2);
                ref_o = ref_w;
            } else {
                fw = ex2(ref_w - ref_o);
            }
        }
        const uint64_t fw2 = f2_pack(fw, fw);
#pragma unroll
        for (int half = 0; half < D / 32; ++half) {
            uint32_t w[32];
            tmem_ld32(lane_addr + grp * 256 + 192 + half * 32, w);
            uint4 raw[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                raw[u] = make_uint4(0u, 0u, 0u, 0u);
                if (ok) raw[u] = staged ? *reinterpret_cast<const uint4 *>(sWinV + sw128_offset(wr, half * 4 + u))
                                        : __ldg(reinterpret_cast<const uint4 *>(vrow + half * 32 + u * 8));
            }
            tmem_wait_ld(w);
            if (half == D / 32 - 1) {           // W of the sweep is in registers: the tensor cores may overwrite it
                tc_fence_before();
                mbar_arrive(&bars[BAR_W_EMPTY + grp]);
            }
            if (ok) {
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t rr[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
#pragma unroll
                    for (int z = 0; z < 4; ++z) {
                        const int x = u * 8 + z * 2;
                        uint64_t &acc = o[half * 16 + (x >> 1)];
                        acc = f2_fma(f2_pack(w[x], w[x + 1]), f2_mul(f2_from_bf16x2(rr[z]), fw2), acc);
                    }
                }
            }
        }
        return true;
    };

    if (staged && !warp_wait(&bars[BAR_WIN_FULL], 0, abort_flag)) return ERR_FWD_OUTPUT;
    if (g.nsw[0] > 0) build_a(0, 0, nullptr, 0);
    if (g.nsw[1] > 0) build_a(1, 0, nullptr, 0);
    for (int k = 0; k < g.nsw[0]; ++k) {
        // the A rows first: the tensor cores wait for them, the W accumulators have a unit's slack
        if (k + 1 < g.nsw[0] && !build_a(0, k + 1, &bars[BAR_A_FREE + 0], k & 1)) return ERR_FWD_OUTPUT;
        if (k + 1 < g.nsw[1] && !build_a(1, k + 1, &bars[BAR_A_FREE + 1], k & 1)) return ERR_FWD_OUTPUT;
        if (!drain(0, k)) return ERR_FWD_OUTPUT;
        if (k < g.nsw[1] && !drain(1, k)) return ERR_FWD_OUTPUT;
    }
    return 0;
}

__device__ __forceinline__ void fwd_rows_sync() { asm volatile("bar.sync 2, 384;" ::: "memory"); }
__device__ __forceinline__ void fwd_out_sync() { asm volatile("bar.sync 3, 128;" ::: "memory"); }

// Merge of the RE partial results of every query row and the store of out and lse.  `buf`: 128 rows of D + 4
// floats, then two rows of 128 statistics (the K1/V1 rows, which nothing reads any more).
template <int D, int RE>
__device__ __forceinline__ void fwd_store(const FwdParams &P, const FwdGeom &g, const float *buf) {
    constexpr int LD = D + 4, RI = TQ / RE, PER = D / RE, VEC = PER < 4 ? PER : 4;      // PER channels of a row per thread
    const KernelParams &kp = P.kp;
    const int r = threadIdx.x & 127, ii = r & (RI - 1), c0 = (r / RI) * PER, i = g.i0 + ii;
    if (i >= kp.n) return;
    __nv_bfloat16 *op = reinterpret_cast<__nv_bfloat16 *>(kp.out.p) + elem_off(kp.out, blockIdx.z, i, blockIdx.y) + c0;
#pragma unroll
    for (int c = 0; c < PER; c += VEC) {
        float x[VEC];
#pragma unroll
        for (int z = 0; z < VEC; ++z) x[z] = 0.f;
#pragma unroll
        for (int s = 0; s < RE; ++s) {
            float v[VEC];
            load_vec<VEC>(buf, (s * RI + ii) * LD + c0 + c, false, v);
#pragma unroll
            for (int z = 0; z < VEC; ++z) x[z] += v[z];
        }
        store_vec<VEC>(op, c, true, x);
    }
}

template <int D, bool SPLIT>
__device__ __forceinline__ void fwd_merge(const FwdParams &P, const FwdGeom &g, const uint64_t (&o)[D / 2], float ref_o,
                                          const float *stats, float *buf, bool bad) {
    constexpr int LD = D + 4;
    const KernelParams &kp = P.kp;
    const int r = threadIdx.x & 127, ii = r & (g.ri - 1), i = g.i0 + ii;
    float *sM = buf + 128 * LD, *sL = sM + 128;
    // the row's two denominators are expressed against their groups' last references, o against ref_o
    const float m0 = stats[768 + r], m1 = stats[896 + r], m = fmaxf(m0, m1);
    const float f0 = m0 > -CUDART_INF_F ? ex2(m0 - m) : 0.f, f1 = m1 > -CUDART_INF_F ? ex2(m1 - m) : 0.f;
    sM[r] = m;
    sL[r] = stats[512 + r] * f0 + stats[640 + r] * f1;
    fwd_out_sync();
    float M = -CUDART_INF_F, L = 0.f;
    for (int s = 0; s < g.re; ++s) M = fmaxf(M, sM[s * g.ri + ii]);
    for (int s = 0; s < g.re; ++s) {
        const float ms = sM[s * g.ri + ii];
        L += ms > -CUDART_INF_F ? sL[s * g.ri + ii] * ex2(ms - M) : 0.f;
    }
    // a CTA in which any wait ran out reports NaN
    const float sc = bad ? CUDART_NAN_F : ref_o > -CUDART_INF_F ? ex2(ref_o - M) / L : 0.f;
#pragma unroll
    for (int x = 0; x < D / 4; ++x) {
        float4 v;
        f2_unpack(o[2 * x], v.x, v.y);
        f2_unpack(o[2 * x + 1], v.z, v.w);
        *reinterpret_cast<float4 *>(buf + r * LD + 4 * x) = make_float4(v.x * sc, v.y * sc, v.z * sc, v.w * sc);
    }
    if (r < g.ri && i < kp.n)       // (lg2.approx would be off by 2e-6 at the denominators of a long window)
        kp.lse[((int64_t)blockIdx.z * kp.hq + blockIdx.y) * kp.n + i] = bad ? CUDART_NAN_F : (M + (SPLIT ? log2f(L) : lg2(L))) * 0.6931471805599453f;
    fwd_out_sync();
    switch (g.re) {
        case 2: fwd_store<D, 2>(P, g, buf); break;
        case 4: fwd_store<D, 4>(P, g, buf); break;
        case 8: fwd_store<D, 8>(P, g, buf); break;
        default: fwd_store<D, 16>(P, g, buf); break;
    }
}

template <int D, bool SPLIT>
__global__ void __launch_bounds__(FWD_THREADS, 1)
fwd_kernel(const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapV,
           const __grid_constant__ CUtensorMap mapK2, const __grid_constant__ CUtensorMap mapV2, const FwdParams P) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = align_smem(smem_raw);
    uint8_t *sK = smem;
    uint8_t *sV = sK + (size_t)max(P.nslots, 3) * FWD_UNIT_BYTES;
    uint8_t *sA = sV + (size_t)max(P.nslots, 3) * FWD_UNIT_BYTES;         // [2] one tile per group
    uint8_t *sWin = sA + 2 * FwdA<D, SPLIT>::BYTES;
    float *stats = reinterpret_cast<float *>(sWin + (size_t)P.win_boxes * 2 * 4096);
    uint64_t *bars = reinterpret_cast<uint64_t *>(stats + FWD_STATS_FLOATS);
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bars + BAR_COUNT);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_holder + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);        // warp-uniform, and known to be
    if (threadIdx.x == 0) {
        for (int x = 0; x < BAR_COUNT; ++x) {
            const bool many = (x >= BAR_P_FULL && x < BAR_P_FULL + 4) || (x >= BAR_W_EMPTY && x < BAR_W_EMPTY + 2) ||
                              (x >= BAR_A_FULL && x < BAR_A_FULL + 2) || (x >= BAR_REF_FULL && x < BAR_REF_FULL + 2);
            const bool two = x <= BAR_WIN_FULL;          // FULL: the two producers; FREE: one commit from each group
            mbar_init(&bars[x], many ? 128u : two ? 2u : 1u);
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
    const FwdGeom g = fwd_geom(P);

    int err = 0;
#ifdef SA2_PROF
    const long long prof_t0 = clock64();
    sa2::sm100::prof_begin();
#endif
    if (warp < 4) {
        reg_dealloc<FWD_REGS_ISSUE>();                // one instruction for the whole warpgroup
        if (warp == 0) err = fwd_mma<D, SPLIT>(P, g, 0, tmem, sK, sV, sA, bars, abort_flag);
        else if (warp == 1) err = fwd_mma<D, SPLIT>(P, g, 1, tmem, sK, sV, sA, bars, abort_flag);
        else if (warp == 2) err = fwd_producer(P, g, &mapK, &mapK2, sK, sWin, bars, abort_flag);
        else err = fwd_producer(P, g, &mapV, &mapV2, sV, sWin + (size_t)P.win_boxes * 4096, bars, abort_flag);
    } else if (warp >= 8) {
        reg_dealloc<FWD_REGS_SOFTMAX>();
        err = fwd_softmax<SPLIT>(P, g, (warp - 8) >> 2, tmem, D, stats, bars, abort_flag);
        // the barrier sits outside fwd_softmax so that a group that gave up still reaches it
        fwd_rows_sync();
    } else {
        reg_alloc<FWD_REGS_OUT>();
        uint64_t o[D / 2];
#pragma unroll
        for (int x = 0; x < D / 2; ++x) o[x] = 0ull;
        float ref_o = -CUDART_INF_F;
        err = fwd_output<D, SPLIT>(P, g, tmem, o, ref_o, sWin, sA, stats, bars, abort_flag);
        fwd_rows_sync();                              // both groups' denominators are in shared memory
        if (err) *abort_flag = 1;
        fwd_merge<D, SPLIT>(P, g, o, ref_o, stats, reinterpret_cast<float *>(sK), err != 0 || *abort_flag != 0);
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
// Query rows per tile.  Measured on a B200: a tile costs ~5500 cycles of set-up, first loads and merge, a 64-key
// unit ~650 cycles while both softmax groups have sweeps and ~1100 when one works alone.  Fewer rows per tile
// mean more tiles with fewer sweeps each (a short or thin problem then fills the chip), more set-up and, below 64
// rows, no fewer units per sweep; the choice is the smallest total over one tile per SM at a time.  The result of
// a batch element must not depend on the others that ride in the call (to the last bit: callers cut batches into
// chunks), so the rule assumes four of them: at one element a tile may be twice as long as it could be, at
// sixteen there may be twice as many tiles as needed.
inline int fwd_ri_log2(const sa2_shape &s, int sms) {
    const double unit = s.d == 128 ? 1.7 : 1.;          // head dim 128: twice the products, streamed
    int best = 6;
    double best_cost = 0.;
    for (int l = 6; l >= 3; --l) {
        const int ri = 1 << l, re = TQ >> l;
        const double tiles = (double)((s.n + ri - 1) / ri) * s.hq * 4.;
        const int rows = ri < s.n ? ri : s.n;
        const int keys = s.w1 + rows - 1 < s.n + s.off1 ? s.w1 + rows - 1 : s.n + s.off1;
        const int units = (keys + FWD_UNIT - 1) / FWD_UNIT;
        const int w2 = s.w2 < s.n + s.off2 ? s.w2 : s.n + s.off2;
        const int sweeps = (w2 + re - 1) / re;
        const double both = sweeps * units * 650. * unit, one = ((sweeps + 1) / 2) * units * 1100. * unit;
        const double waves = tiles > sms ? tiles / sms : 1.;
        const double cost = waves * (5500. + (both > one ? both : one));
        if (l == 6 || cost < 0.98 * best_cost) { best = l; best_cost = cost; }
    }
    return best;
}
inline int fwd_win_boxes(int w2, int ri_log2) {
    const int rows = w2 + (1 << ri_log2) - 1;
    return rows <= FWD_WIN_ROWS ? (rows + 31) / 32 : 0;
}
// slots for the widest window of a tile, or as many as fit beside everything else
inline int fwd_slots(int w1, int ri_log2, int win_boxes, int a_tiles) {
    const int units = (w1 + (1 << ri_log2) - 1 + FWD_UNIT - 1) / FWD_UNIT;
    const size_t fixed = 1024 + (size_t)win_boxes * 8192 + a_tiles * TILE_BYTES + FWD_STATS_FLOATS * 4 + BAR_COUNT * 8 + 64;
    const int room = (int)((232448 - fixed) / (2 * FWD_UNIT_BYTES)), most = room < FWD_MAX_SLOTS ? room : FWD_MAX_SLOTS;
    return units < most ? units : most;
}

}  // namespace tc
}  // namespace sa2
