// Backward kernel for dQ, dK2, dV2 on tcgen05 tensor cores (bf16 operands,
// fp32 accumulation in TMEM, head dims 32, 64 and 128), plus the reduction of its
// partials and of those of dK1 / dV1.
//
// A tile is 128 (query row, offset) pairs of one (batch, query head), e = i - k being the offset.  PAIR: 64 query rows i times two
// consecutive offsets; rows 0-63 have the even offset of a "sweep", rows 64-127 the odd one.  Otherwise 128 query rows and one offset
// a sweep (head dims 32 and 64; bq_plan chooses).  A CTA owns the query rows and a
// subset ("split") of their K1/V1 units and offsets.  Because the backward recomputes probabilities from the saved
// logsumexp, the splits of one query tile are independent; each writes fp32 partials to scratch and a small second kernel
// adds them in a fixed order (splits, then the query heads of a kv group), so results are reproducible.
// Head dims 32 and 64: a split keeps its 64-key units (at most nine, or six beside 128 rows) resident in shared memory; with pairs a
// window of up to 513 keys is one split.  Head dim 128: the units stream through a three-slot TMA ring (32 KB per slot), once per sweep, from L2: a slot is
// refilled when the U / W products of its unit are done.  The offsets may be split as well (bq_split).
//
// Why pairs: in long windows the window of 64 rows is w1 + 63 keys where that of 128 rows is w1 + 127 (9 units against 10 at w1 = 512), it
// fits the shared memory of one CTA, so that dQ needs no partials, and a sweep's operands and its fold are shared by 9 units
// where a window in two splits shared them by 4 and 6.  Why not always: a sweep takes at least what its fold takes, ~5300 cycles with
// pairs (their fold has a hand-over in the middle) against ~2900 and ~790 for each unit with 128 rows.
//
// SPLIT (head dim 32, and second windows above 56 rows: see bq_plan) keeps A_e, B_e, P and G as a bf16 value and a bf16 rest
// each, with twice the products; the rests cost two units at head dim 64 (of nine or six) and two of the three ring slots at 128.
//
// Per sweep the fold groups form A[r] = q_i * k2_{i-e} and B[r] = dO_i * v2_{i-e}; per 64-key
// unit the tensor cores compute
//     S = A K1^T      dP = B V1^T                     (rows r, columns j)
// the compute warps (one thread per row and half of the unit's columns) form
//     P = exp2(c S - lse2_i)     G = P * (dP - D_i)    (bf16, back into TMEM)
// and the tensor cores accumulate over the sweep
//     U += G K1       W += P V1                       (K1/V1 as MN-major B)
// At the end of a sweep the row owners fold U, W into
//     dQ_i += U * k2_{i-e}                             (registers; the two rows of a query are added at the end)
//     dK2_{i-e} += U * q_i,  dV2_{i-e} += W * dO_i     (fp32 rows in shared memory)
// With pairs both rows (i, e) and (i + 1, e + 1) add to row i - e of the shared accumulators: the even rows of the sweep do their first
// half of the channels while the odd rows do the second one, a barrier, and then the other halves, so that each value has one writer
// at a time and a fixed order.  65 rows are live in a sweep and the next one starts two rows further down (without pairs 128, and one):
// the accumulators are a ring of as many rows, and whoever adds to a row last writes it to the slab in global memory instead.
//
// Warps (640 threads): 0 issuer of U (after loading the units; head dim 128: of U and W); 1 TMEM owner and issuer of
// S; 2 issuer of dP; 3 issuer of W (head dim 128: TMA producer of the ring); 4-7 and 8-11 two compute groups, each
// forming 32 of the 64 columns of every unit (P, G); 12-15 form A of the next sweep
// and fold U of the last one into dQ / dK2, 16-19 do the same with B, W and dV2.
// TMEM columns: S / dP buffer x -> S/P [128x, 128x+64), dP/G [128x+64, 128x+128); P and G (bf16, 16 columns per
// 32 keys; with SPLIT their rests in the next 16) overwrite the S and dP columns of the same keys - columns that the
// writing compute group has itself read - so a buffer is busy from the issue of S / dP until the U / W products of its unit are
// done.  Up to head dim 64 three such buffers are in flight (issue, compute and U / W of different units overlap), U [384, 448) and
// W [448, 512); head dim 128 has two buffers, U [256, 384) and W [384, 512).  The fold groups read U / W into registers before the
// next sweep's first product.
//
// Bound, up to head dim 64: the compute groups, busy ~1080 of ~1280 cycles a unit (512 of them MUFU cycles of two warps a scheduler;
// the wait accounting shows them waiting 10 to 15 % of the time, every other role half of it).  Everything that goes through shared
// memory waits behind the tensor cores' operand fetches (300 cycles and more an access), so a fold reads half a row of U or W at a
// time, loads what two pieces of it need before it adds and stores, and has its second keys in a staged copy; windows of few units
// are bound by the folds, ~6000 cycles a sweep.  At head dim 128 the fold of U has no registers for half a row: its ~18000 cycles a
// sweep (operands from L2, half a row per lane) hold up the next sweep's U / W.
// Measured, this kernel and its reduction, against tiles of 128 rows and one offset with the window in two splits (head dim 64) or two
// CTAs of 64 channels each that formed S and dP twice (head dim 128): b4 n4096 h8 d64 w512/32 1.66 -> 1.40 ms, b1 n3001 h8 w1024/16
// 293 -> 285 us, b4 n1966 h4 w105/26 188 -> 182, b1 n300 h4 w300/32 38 -> 27, b1 n16384 h16 d128 w512/32 8.74 -> 7.4 ms.
// SPLIT: b4 n3000 h8 d32 w512/32 1.42 -> 1.13 ms, d64 w512/64 4.53 -> 4.24, d128 w512/64 16.7 -> 10.4 (both chunks of a group's columns read
// before either is written, as it was at first, does not fit 80 registers: 2.12, 5.59 and 12.2).
// Tiles of 128 rows, this kernel's (in brackets: an earlier one's, with all accumulator rows and no staged second keys) against pairs: b128
// n128 h8 d64 w512/32 583 (644) / 802 us, b16 n128 h8 89 (100) / 113, b4 n3000 h8 d64 w64/9 217 (231) / 254, w76/10 247 (253) / 267,
// b64 n256 hq8 hk4 725 (755) / 869, b128 n128 h8 d32 530 (543) / 675.
// Measured and not kept (head dim 64, C = b4 n4096 above, S = b4 n1966): a row of U or W read at once, which frees the accumulators
// sooner and leaves no registers to load ahead, C 1.35 but S 229 us; U and W read sixteen channels at a time, C 1.87; compute groups on
// alternate units, C 1.40; 32 columns at a time with 88 registers, C 1.46; the next sixteen columns fetched ahead, C 1.74 (spills); the
// mask applied to every unit, C 1.42.  Head dim 128: a ring of two slots with q and dO staged in its place 8.8 ms, one slot 10.5,
// eight channels at a time with operands fetched one to four ahead 7.9 to 8.2, both operands built by the W fold 7.8.
#pragma once
#include "sa2_tc_bwd_k1.cuh"

namespace sa2 {
namespace tc {

__host__ __device__ constexpr int bq_rows(bool pair) { return pair ? 64 : 128; }      // query rows of a tile
__host__ __device__ constexpr int bq_step(bool pair) { return pair ? 2 : 1; }         // offsets of a sweep
constexpr int BQ_FINE_W2 = 56;   // second windows above this keep fp32 accuracy (bq_plan)
// Most offsets of a CTA: the second keys they pair with are staged in shared memory up to head dim 64.  (The wait accounting wants
// some of it, and a ring slot of head dim 128.)
#ifdef SA2_PROF
constexpr bool BQ_ACCOUNTED = true;
constexpr int BQ_MAX_EPC = 40;
#else
constexpr bool BQ_ACCOUNTED = false;
constexpr int BQ_MAX_EPC = 56;
#endif

// Register hand-over between warpgroups.  A group can only grow by what another has released, or its setmaxnreg
// never returns, so the budgets must add up to what the block was launched with: five groups of 96 (640 threads).  Up to head dim
// 64 the U fold takes 176 (dQ, the q row and half a row of U, 128 registers, and what two pieces need), the W fold 112; at head dim 128 the U fold 184 (dQ,
// 128 registers, and chunks of the rest), the W fold 96.
template <int D, bool SPLIT, bool PAIR = true> struct BqCfg {
    static constexpr int THREADS = 640;
    static constexpr int ROWS = bq_rows(PAIR), STEP = bq_step(PAIR), RING = PAIR ? 65 : 128;        // RING: rows of the shared accumulators
    static constexpr int REGS_LAUNCH = 96, REGS_ISSUE = D <= 64 ? 32 : 40, REGS_COMPUTE = 80;
    static constexpr int REGS_FOLD = D <= 64 ? 176 : 184, REGS_FOLD_W = D <= 64 ? 112 : 96;
    static_assert(REGS_COMPUTE <= REGS_LAUNCH, "the compute groups release registers");
    static_assert(REGS_ISSUE + 2 * REGS_COMPUTE + REGS_FOLD + REGS_FOLD_W == THREADS / 128 * REGS_LAUNCH, "register pool must balance");
    static constexpr int CB = D == 128 ? 2 : 1;                  // 64-channel blocks of a row
    static constexpr int KSTEPS = D / 16;                        // K = 16 steps of S and dP
    static constexpr uint32_t BLK = 128 * 128;                   // A / B: one [128 rows][64 channels] swizzled block
    // SPLIT: A, B, P and G are each a bf16 value and a bf16 rest.  The rests of A / B fill the free half of the rows
    // at head dim 32 and take blocks of their own otherwise, for which K1 / V1 make room
    static constexpr uint32_t REST = D == 32 ? 64 : CB * BLK;    // bytes from an element of A / B to its rest
    static constexpr uint32_t TILE = CB * BLK * (SPLIT && D > 32 ? 2 : 1);        // A or B
    static constexpr uint32_t UBLK = 8192;                       // one channel block of a 64-row unit of K1 / V1
    static constexpr int MAX_UNITS = SPLIT && D == 64 ? (PAIR ? 7 : 4) : (PAIR ? 9 : 6);   // resident units of a split (head dims 32, 64)
    static constexpr int NSLOT = SPLIT ? 1 : BQ_ACCOUNTED ? 2 : 3;                  // ring slots (head dim 128)
    static constexpr uint32_t KV_BYTES = D <= 64 ? MAX_UNITS * UBLK : NSLOT * 2 * UBLK;
    static constexpr int NBUF = D <= 64 ? 3 : 2;                 // S / dP (P / G) buffers in TMEM
    static constexpr uint32_t U0 = NBUF * 128, W0 = U0 + (D == 128 ? 128 : 64);      // TMEM columns of U and W
    // Shared accumulators of dK2 / dV2: rows of D + 4 floats, so that the row-per-thread accesses of a warp spread over all banks
    // and the offsets inside a row are compile-time constants; head dim 128 has no room for the padding and XORs the
    // 16-byte chunk with the row instead.
    static constexpr int ACC_STRIDE = D == 128 ? 128 : D + 4;
    static constexpr uint32_t ACC_BYTES = RING * ACC_STRIDE * 4;
    // Up to head dim 64 the second keys of the tile, which the U fold reads a row per lane: that costs the L1 32 cycles an
    // instruction from global memory and four from here.
    static constexpr bool STAGE_Y = D <= 64;
    static constexpr uint32_t STAGE_BYTES = STAGE_Y ? (ROWS - 1 + BQ_MAX_EPC) * 128 : 0;
    static constexpr size_t SMEM = 1024 + 2 * (size_t)KV_BYTES + 2 * TILE + 2 * ACC_BYTES + STAGE_BYTES + 256;
    static_assert(SMEM <= 227 * 1024, "shared memory of an SM");
};

// Entry 0 of a pair belongs to A, S, U and entry 1 to B, dP, W, except S_FULL ... G_DONE.
enum BqBar {
    BQ_KV_FULL = 0,
    BQ_AB_FULL = 1,      // [2]
    BQ_AB_EMPTY = 3,     // [2]
    BQ_S_FULL = 5,       // [3] per buffer
    BQ_P_FULL = 8,       // [3]
    BQ_G_DONE = 11,      // [3] the U / W products of the buffer's unit have completed
    BQ_W_FULL = 14,      // [2]
    BQ_W_EMPTY = 16,     // [2] the fold group holds the accumulator of the sweep in registers
    BQ_KV_SLOT = 18,     // [3] head dim 128: the K1/V1 unit of the ring slot has landed
    BQ_KV_FREE = 21,     // [3] head dim 128: the U / W products that read the slot have completed
    BQ_FOLD_MID = 24,    // [2] every fold thread has added the first half of its channels
    BQ_FOLD_SYNC = 26,   // [2] every fold thread has added its sweep into the shared accumulators
    BQ_BAR_COUNT = 28
};

enum { ERR_BQ_PRODUCER = 256, ERR_BQ_MMA = 512, ERR_BQ_COMPUTE = 1024, ERR_BQ_BUILDER = 2048 };

struct BqParams {
    KernelParams kp;
    float c;            // scale * log2(e)
    int nu;             // 64-key units of a query tile's window
    int nsplit;         // CTAs sharing one query tile: tsplit x (offset splits)
    int tsplit;         // splits of the K1/V1 window
    int units_per_split;
    int epc;            // second-key offsets of a CTA, a multiple of those of a sweep: split s takes [epc * (s / tsplit), +epc)
    int nqt;            // query tiles
    float *part_dq;     // [nsplit][b][n][hq][d]
    float *part_k2;     // [b][hq][nqt][nsplit][2][rows of a tile - 1 + epc][d]   (dK2 slab, then dV2 slab)
    int *status;
    // what the reduction adds up: dQ and dK2/dV2, and the dK1/dV1 partials of ce CTAs per key tile
    const float *part_k1;
    int ce, reduce_q, reduce_k1;
};

// (a query tile with one split writes dQ itself and needs no partials)
inline size_t bq_part_dq_bytes(const sa2_shape &s, int nsplit) { return nsplit == 1 ? 0 : (size_t)nsplit * s.b * s.n * s.hq * s.d * sizeof(float); }
inline size_t bq_part_k2_bytes(const sa2_shape &s, int rows, int nsplit, int epc) {
    const size_t nqt = (s.n + rows - 1) / rows;
    return (size_t)s.b * s.hq * nqt * nsplit * 2 * (rows - 1 + epc) * s.d * sizeof(float);
}

struct BqGeom {
    int qt, split;               // query tile and split of this CTA
    int i0;
    int e0, e1;                  // its offsets; sweep t: e0 + 2 t and the one behind it (or e0 + t)
    int nsweeps;
    int ubase;                   // first-key row of the CTA's unit 0; unit x covers rows ubase + 64 x ... + 63
    int nunits;                  // 64-key units the CTA visits in every sweep
    int total;                   // nunits * nsweeps
};

template <bool PAIR>
__device__ __forceinline__ BqGeom bq_geom(const BqParams &P, int qt, int split) {
    BqGeom g;
    const KernelParams &kp = P.kp;
    g.qt = qt;
    g.split = split;
    constexpr int ROWS = bq_rows(PAIR), STEP = bq_step(PAIR);
    g.i0 = qt * ROWS;
    const int i_last = min(g.i0 + ROWS - 1, kp.n - 1);
    g.e0 = (split / P.tsplit) * P.epc;
    g.e1 = min(min(kp.w2, g.e0 + P.epc), i_last + kp.off2 + 1);
    g.nsweeps = max(0, (g.e1 - g.e0 + STEP - 1) / STEP);
    const int ts = split % P.tsplit;
    const int base = g.i0 + kp.off1 + ROWS - 64 * P.nu;       // unit x of the window covers rows base + 64 x ...
    const int first = base >= 0 ? 0 : min(P.nu - 1, (-base) / 64);
    const int begin = max(first, ts * P.units_per_split), end = min(P.nu, (ts + 1) * P.units_per_split);
    g.ubase = base + 64 * begin;
    g.nunits = max(0, end - begin);
    g.total = g.nunits * g.nsweeps;
    return g;
}

// ---------------------------------------------------------------- issuers of S (warp 1) and dP (warp 2)
// Unit u (numbered over the whole kernel) is unit u % nunits of sweep u / nunits and uses TMEM buffer u % NBUF.
// A warp issues about one tcgen05.mma per 45-90 cycles, so the two product stages have an issuing warp
// each; U / W are accumulated by one warp only, which keeps the summation order fixed.
// which = 0: S = A K1^T into columns [128 buf, +64); which = 1: dP = B V1^T into [128 buf + 64, +64).
template <int D, bool SPLIT>
__device__ __forceinline__ int bq_mma_first(const BqGeom &g, int which, uint32_t tmem, uint8_t *sKV, uint8_t *sAB,
                                            uint64_t *bars, volatile int *abort_flag) {
    using C = BqCfg<D, SPLIT>;
    constexpr uint32_t IDESC_F = idesc_bf16(128, 64, false, false);
    const uint64_t dT = smem_desc_sw128(smem_u32(sKV)), dA = smem_desc_sw128(smem_u32(sAB));
    if constexpr (D <= 64) {
        if (!mbar_wait_warp(&bars[BQ_KV_FULL], 0, abort_flag)) return ERR_BQ_MMA;
    }
    int u = 0, buf = 0, use = 0;                         // use = u / NBUF: how often the buffer has been used before
    int slot = 0, suse = 0;                              // head dim 128: ring slot u % NSLOT and u / NSLOT
    for (int t = 0; t < g.nsweeps; ++t) {
        if (!mbar_wait_warp(&bars[BQ_AB_FULL + which], t & 1, abort_flag, 0, 1)) return ERR_BQ_MMA;
        for (int w = 0; w < g.nunits; ++w, ++u) {
            // the buffer holds P / G of its previous unit until the U / W products of that unit are done
            if (use >= 1 && !mbar_wait_warp(&bars[BQ_G_DONE + buf], (use - 1) & 1, abort_flag, 0, 2)) return ERR_BQ_MMA;
            if constexpr (D == 128) {
                if (!mbar_wait_warp(&bars[BQ_KV_SLOT + slot], suse & 1, abort_flag, 0, 3)) return ERR_BQ_MMA;
            }
            tc_fence_after();
            if (elect_one()) {
                const uint32_t d = tmem + buf * 128 + which * 64;
                const uint64_t kt = dT + (uint64_t)((D <= 64 ? w * C::UBLK : slot * 2 * C::UBLK) >> 4);
#pragma unroll
                for (int k = 0; k < (SPLIT ? 2 : 1) * C::KSTEPS; ++k) {
                    const int rest = k / C::KSTEPS, x = k % C::KSTEPS, cb = x >> 2;        // K = 16 step x of 64-channel block cb
                    mma_ss(d, dA + ((rest * C::REST + cb * C::BLK) >> 4) + 2 * (x & 3), kt + ((cb * C::UBLK) >> 4) + 2 * (x & 3), IDESC_F, k > 0);
                }
                tc_commit(&bars[BQ_S_FULL + buf]);
            }
            if (++buf == C::NBUF) { buf = 0; ++use; }
            if (++slot == C::NSLOT) { slot = 0; ++suse; }
        }
        if (elect_one()) tc_commit(&bars[BQ_AB_EMPTY + which]);
    }
    return 0;
}

// ---------------------------------------------------------------- head dim 128: TMA producer of the K1/V1 ring (warp 3)
template <int D, bool SPLIT>
__device__ __forceinline__ int bq_ring_producer(const BqParams &P, const BqGeom &g, const CUtensorMap *mapK, const CUtensorMap *mapV,
                                                uint8_t *sK, uint8_t *sV, uint64_t *bars, volatile int *abort_flag) {
    using C = BqCfg<D, SPLIT>;
    const int hk = blockIdx.y / P.kp.g;
    prefetch_tmap(mapK);
    prefetch_tmap(mapV);
    int w = 0, slot = 0, suse = 0;
    for (int u = 0; u < g.total; ++u) {
        // the slot is free when the U / W products of the unit it held are done
        if (suse >= 1 && !mbar_wait_warp(&bars[BQ_KV_FREE + slot], (suse - 1) & 1, abort_flag, 32, 1)) return ERR_BQ_PRODUCER;
        const int row = g.ubase + 64 * w;
        if (elect_one()) {
            mbar_arrive_expect_tx(&bars[BQ_KV_SLOT + slot], 4 * C::UBLK);
#pragma unroll
            for (int cb = 0; cb < 2; ++cb) {
                tma_load_4d(sK + slot * 2 * C::UBLK + cb * C::UBLK, mapK, &bars[BQ_KV_SLOT + slot], cb * 64, hk, row, blockIdx.z);
                tma_load_4d(sV + slot * 2 * C::UBLK + cb * C::UBLK, mapV, &bars[BQ_KV_SLOT + slot], cb * 64, hk, row, blockIdx.z);
            }
        }
        if (++w == g.nunits) w = 0;
        if (++slot == C::NSLOT) { slot = 0; ++suse; }
    }
    // every load must have landed before the CTA may exit, even if the consumers gave up
    for (int u = max(0, g.total - C::NSLOT); u < g.total; ++u)
        if (!mbar_wait_warp(&bars[BQ_KV_SLOT + u % C::NSLOT], (u / C::NSLOT) & 1, abort_flag, 32)) return ERR_BQ_PRODUCER;
    return 0;
}

// ---------------------------------------------------------------- issuers of U, W
// part 0 (warp 0; up to head dim 64, after loading the units): U += G K1; part 1 (warp 3): W += P V1; part 2 (head dim
// 128, warp 0, whose N = 128 products keep the pipe busy from one warp): both.  Each accumulator has one issuing warp, which
// keeps its summation order fixed.
template <int D, bool SPLIT>
__device__ __forceinline__ int bq_mma_second(const BqParams &P, const BqGeom &g, int part, const CUtensorMap *mapK, const CUtensorMap *mapV,
                                             uint32_t tmem, uint8_t *sK, uint8_t *sV, uint64_t *bars, volatile int *abort_flag) {
    using C = BqCfg<D, SPLIT>;
    constexpr uint32_t IDESC_G = idesc_bf16(128, D, false, true);
    if constexpr (D <= 64) {
        if (part == 0) {
            const int hk = blockIdx.y / P.kp.g;
            prefetch_tmap(mapK);
            prefetch_tmap(mapV);
            if (elect_one()) {
                mbar_arrive_expect_tx(&bars[BQ_KV_FULL], 2 * C::UBLK * g.nunits);
                for (int t = 0; t < g.nunits; ++t) {
                    const int row = g.ubase + 64 * t;
                    tma_load_4d(sK + (size_t)t * C::UBLK, mapK, &bars[BQ_KV_FULL], 0, hk, row, blockIdx.z);
                    tma_load_4d(sV + (size_t)t * C::UBLK, mapV, &bars[BQ_KV_FULL], 0, hk, row, blockIdx.z);
                }
            }
        }
        if (!mbar_wait_warp(&bars[BQ_KV_FULL], 0, abort_flag)) return ERR_BQ_PRODUCER;
    }
    // head dim 128: N = 128, the channel blocks of a unit 8 KB apart
    const uint64_t dK = smem_desc_sw128(smem_u32(sK), 1024, D == 128 ? C::UBLK : 16), dV = smem_desc_sw128(smem_u32(sV), 1024, D == 128 ? C::UBLK : 16);
    int u = 0, buf = 0, use = 0, slot = 0;
    for (int t = 0; t < g.nsweeps; ++t) {
        for (int w = 0; w < g.nunits; ++w, ++u) {
            if (!mbar_wait_warp(&bars[BQ_P_FULL + buf], use & 1, abort_flag, 0, 1)) return ERR_BQ_MMA;
            // the fold groups must have read the accumulators of the last sweep
            if (w == 0 && t >= 1) {
                if (part != 1 && !mbar_wait_warp(&bars[BQ_W_EMPTY], (t - 1) & 1, abort_flag, 0, 2)) return ERR_BQ_MMA;
                if (part != 0 && !mbar_wait_warp(&bars[BQ_W_EMPTY + 1], (t - 1) & 1, abort_flag, 0, 2)) return ERR_BQ_MMA;
            }
            tc_fence_after();
            const uint64_t off = (uint64_t)((D <= 64 ? w * C::UBLK : slot * 2 * C::UBLK) >> 4);
            const uint32_t a = tmem + buf * 128;
            if (elect_one()) {
                // keys [32 x, +32) of G are 16 columns at 64 + 32 x, those of P at 32 x; with SPLIT their rests behind them
#pragma unroll
                for (int k = 0; k < (SPLIT ? 8 : 4); ++k) {
                    const uint32_t col = (k & 2) * 16 + (k & 1) * 8 + (k >> 2) * 16;
                    if (part != 1) mma_ts(tmem + C::U0, a + 64 + col, dK + off + 128 * (k & 3), IDESC_G, w + k > 0);
                    if (part != 0) mma_ts(tmem + C::W0, a + col, dV + off + 128 * (k & 3), IDESC_G, w + k > 0);
                }
                tc_commit(&bars[BQ_G_DONE + buf]);
                if constexpr (D == 128) tc_commit(&bars[BQ_KV_FREE + slot]);
            }
            if (++buf == C::NBUF) { buf = 0; ++use; }
            if (++slot == C::NSLOT) slot = 0;
        }
        if (elect_one()) {
            if (part != 1) tc_commit(&bars[BQ_W_FULL]);
            if (part != 0) tc_commit(&bars[BQ_W_FULL + 1]);
        }
    }
    return 0;
}

// ---------------------------------------------------------------- compute (warps 4-7 and 8-11): P and G
// P and G = P (dP - D) of two columns, as packed bf16.  The kernel's issue slots count here (728 warp instructions a unit
// and scheduler before the packed arithmetic of this and of the folds), so two columns share an instruction.
// SPLIT: and what the rounding left of each.
template <bool SPLIT>
__device__ __forceinline__ void pg_pair(float p0, float p1, uint32_t dp0, uint32_t dp1, uint64_t ndl2, uint32_t &pp, uint32_t &gg, uint32_t &pr,
                                        uint32_t &gr) {
    float g0, g1;
    f2_unpack(f2_mul(f2_pack(p0, p1), f2_add(f2_pack(dp0, dp1), ndl2)), g0, g1);
    pp = pack_bf16(p0, p1);
    gg = pack_bf16(g0, g1);
    if constexpr (SPLIT) {
        pr = pack_rest(p0, p1, pp);
        gr = pack_rest(g0, g1, gg);
    }
}
// Group cg forms columns [32 cg, +32) of every unit, which halves the time between S / dP and P / G.
template <int D, bool SPLIT, bool PAIR>
__device__ __forceinline__ int bq_compute(const BqParams &P, const BqGeom &g, int cg, uint32_t tmem, uint64_t *bars, volatile int *abort_flag) {
    using C = BqCfg<D, SPLIT, PAIR>;
    const KernelParams &kp = P.kp;
    const int r = threadIdx.x & 127;                  // row of the tile = TMEM lane
    const uint32_t lane_addr = tmem + ((uint32_t)(r & 96) << 16);
    const int h = blockIdx.y, b = blockIdx.z;
    const int i = g.i0 + (r & (C::ROWS - 1));
    const bool row_ok = i < kp.n;
    const float c = P.c;
    float lse2 = 0.f, dl = 0.f;
    if (row_ok) {
        const int64_t o = ((int64_t)b * kp.hq + h) * kp.n + i;
        lse2 = kp.lse[o] * 1.4426950408889634f;
        dl = kp.delta[o];
    }
    const uint64_t c2 = f2_pack(c, c), nlse2 = f2_pack(-lse2, -lse2), ndl2 = f2_pack(-dl, -dl);
    const int c0 = 32 * cg;                           // the group's first column
    int e = g.e0 + (PAIR ? r >> 6 : 0), w = 0;
    for (int u = 0; u < g.total; ++u, ++w) {
        if (w == g.nunits) { w = 0; e += C::STEP; }
        const bool sweep_ok = row_ok && e < g.e1 && i + kp.off2 - e >= 0;
        const int buf = u % C::NBUF, use = u / C::NBUF;
        const int j0 = g.ubase + 64 * w;
        const int d1 = i + kp.off1 - j0;
        const int hi = sweep_ok ? min(d1, 63) : -1;         // valid columns: lo < col <= hi
        const int lo = max(d1 - kp.w1, -j0 - 1);
        // valid columns are the integers in (lo, hi]: 2048 (half + 1/2 - |col - mid|) is at least 1024
        // inside and at most -1024 outside, so the minimum with it leaves the exponents of valid cells
        // alone and makes P exactly 0 elsewhere, whatever S is there (FMA pipe instead of compares and
        // selects on the ALU pipe; all values are exact)
        const float mid = 1024.f * (float)(lo + 1 + hi), half = 1024.f * (float)(hi - lo);
        const uint32_t s_addr = lane_addr + buf * 128, d_addr = s_addr + 64;
        if (!warp_wait(&bars[BQ_S_FULL + buf], use & 1, abort_flag, 1)) return ERR_BQ_COMPUTE;
        tc_fence_after();
        const bool full = __all_sync(0xffffffffu, lo < 0 && hi >= 63);
        // sixteen columns at a time.  P / G go over the first half of the group's columns of S / dP (the other group's columns of the
        // buffer may still be unread), the rests over the second half once that has been read
        uint32_t pr[2][8], gr[2][8];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int col = c0 + 16 * x;
            uint32_t s[16], d[16], pp[8], gg[8];
            tmem_ld16(s_addr + col, s);
            tmem_ld16(d_addr + col, d);
            tmem_wait_ld(s);
            tmem_wait_ld(d);
            if constexpr (SPLIT) {
                if (x == 1) {
                    tmem_st8(s_addr + c0 + 16, pr[0]);
                    tmem_st8(d_addr + c0 + 16, gr[0]);
                }
            }
            auto pass = [&](bool masked) {
                const float m = mid - 2048.f * (float)col;
#pragma unroll
                for (int z = 0; z < 16; z += 2) {
                    float a0, a1;
                    f2_unpack(f2_fma(f2_pack(s[z], s[z + 1]), c2, nlse2), a0, a1);
                    if (masked) {
                        a0 = fminf(a0, half - fabsf(2048.f * z - m));
                        a1 = fminf(a1, half - fabsf(2048.f * (z + 1) - m));
                    }
                    pg_pair<SPLIT>(ex2(a0), ex2(a1), d[z], d[z + 1], ndl2, pp[z >> 1], gg[z >> 1], pr[x][z >> 1], gr[x][z >> 1]);
                }
            };
            if (full) pass(false);
            else if (__all_sync(0xffffffffu, hi < col || lo >= col + 15)) {        // no row of this warp has a valid column here
#pragma unroll
                for (int z = 0; z < 8; ++z) pp[z] = gg[z] = pr[x][z] = gr[x][z] = 0u;
            } else pass(true);
            tmem_st8(s_addr + c0 + 8 * x, pp);
            tmem_st8(d_addr + c0 + 8 * x, gg);
            if constexpr (SPLIT) {
                if (x == 1) {
                    tmem_st8(s_addr + c0 + 24, pr[1]);
                    tmem_st8(d_addr + c0 + 24, gr[1]);
                }
            }
        }
        tmem_wait_st();
        tc_fence_before();
        mbar_arrive(&bars[BQ_P_FULL + buf]);
    }
    return 0;
}

// ---------------------------------------------------------------- fold: U, W -> dQ, dK2, dV2
// (which: the fold group of U, or that of W)
__device__ __forceinline__ void bq_fold_sync(int which) { asm volatile("bar.sync %0, 128;" ::"r"(1 + which) : "memory"); }

__device__ __forceinline__ uint4 mul_bf16x8(const uint4 &x, const uint4 &y) {
    return make_uint4(mul_bf16x2(x.x, y.x), mul_bf16x2(x.y, y.y), mul_bf16x2(x.z, y.z), mul_bf16x2(x.w, y.w));
}

// WHICH = 0 forms A = q_i * k2_{i-e} and folds U into dQ_i (registers) and dK2_{i-e}; WHICH = 1 forms B = dO_i * v2_{i-e} and folds
// W into dV2_{i-e}.  One thread per row of the tile.  Channels are numbered from the half that the row adds first: channel x of
// an odd row is channel x ^ (D / 2) of the tensors.
// Up to head dim 64 the row of q (dO) stays in registers.  At head dim 128 an operand row is fetched by sixteen lanes, 16 bytes each, so
// that a load of the warp is whole rows: with a row per lane every load touched 32 cache lines, ~8000 cycles of L1 a sweep.
template <int D, bool SPLIT, bool PAIR, int WHICH>
__device__ __forceinline__ int bq_fold_body(const BqParams &P, const BqGeom &g, uint32_t tmem, float *acc, uint8_t *sOp, uint8_t *sStage, float *slab, uint64_t (&dq)[D / 2],
                                            uint64_t *bars, volatile int *abort_flag) {
    using C = BqCfg<D, SPLIT, PAIR>;
    constexpr int ROWS = C::ROWS, STEP = C::STEP;
    const KernelParams &kp = P.kp;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = threadIdx.x & 127, odd = PAIR ? __shfl_sync(0xffffffffu, r >> 6, 0) : 0;     // row of the tile = TMEM lane
    const int rot = odd ? D / 2 : 0;
    const uint32_t cols = tmem + ((uint32_t)(r & 96) << 16) + (WHICH ? C::W0 : C::U0);
    const int h = blockIdx.y, b = blockIdx.z, hk = h / kp.g;
    const int ir = r & (ROWS - 1), i = g.i0 + ir;
    const bool row_ok = i < kp.n;
    constexpr int NC = D / 8;                         // 16-byte chunks of a row
    constexpr bool HELD = D <= 64;                    // the row of q (dO) stays in registers
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const TensorRef &tx = WHICH ? kp.dout : kp.q, &ty = WHICH ? kp.v2 : kp.k2;
    const uint4 *xrow = reinterpret_cast<const uint4 *>(reinterpret_cast<const __nv_bfloat16 *>(tx.p) + elem_off(tx, b, row_ok ? i : 0, h));
    uint4 xr[HELD ? NC : 1];
    if constexpr (HELD) {
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) xr[cc] = row_ok ? __ldg(xrow + (cc ^ (rot / 8))) : zero;
    }
    const __nv_bfloat16 *ybase = reinterpret_cast<const __nv_bfloat16 *>(ty.p) + elem_off(ty, b, 0, hk);
    if constexpr (WHICH == 0) {
#pragma unroll
        for (int x = 0; x < D / 2; ++x) dq[x] = 0;
    }
    constexpr bool STAGE_Y = C::STAGE_Y && WHICH == 0;
    const int top_row = ir + P.epc - 1 - odd;         // row of the slab, and of the staged second keys, in sweep 0
    auto stage = [&]() {
        const int k0 = g.i0 + kp.off2 - g.e0 - (P.epc - 1);
        for (int x = r; x < (ROWS - 1 + P.epc) * NC; x += 128) {
            const int row = x / NC, cc = x % NC, k = k0 + row;
            *reinterpret_cast<uint4 *>(sStage + sw128_offset(row, cc)) =
                k >= 0 && k < kp.nk2 ? __ldg(reinterpret_cast<const uint4 *>(ybase + (int64_t)k * ty.sn) + cc) : zero;
        }
        bq_fold_sync(WHICH);
    };
    auto ystaged = [&](int t, int cc) { return *reinterpret_cast<const uint4 *>(sStage + sw128_offset(top_row - STEP * t, cc)); };
    auto yrow = [&](int t, bool &ok) {
        const int e = g.e0 + STEP * t + odd, kk = i + kp.off2 - e;
        ok = row_ok && e < g.e1 && kk >= 0;
        return reinterpret_cast<const uint4 *>(ybase + (int64_t)(ok ? kk : 0) * ty.sn);
    };
    auto build_held = [&](int t) -> bool {
        bool ok;
        const uint4 *py = yrow(t, ok);
        uint4 y[NC];
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
            if (STAGE_Y && t > 0) y[cc] = ystaged(t, cc ^ (rot / 8));
            else y[cc] = ok ? __ldg(py + (cc ^ (rot / 8))) : zero;
        }
        if constexpr (!SPLIT) {
#pragma unroll
            for (int cc = 0; cc < NC; ++cc) y[cc] = ok ? mul_bf16x8(xr[HELD ? cc : 0], y[cc]) : zero;
        }
        if (t >= 1 && !warp_wait(&bars[BQ_AB_EMPTY + WHICH], (t - 1) & 1, abort_flag, 3)) return false;
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
            const int pc = cc ^ (rot / 8);
            uint8_t *dst = sOp + sw128_offset(r, pc);
            if constexpr (SPLIT) {       // (formed here: a row of products and one of rests would not fit the registers)
                const uint4 hi = ok ? mul_bf16x8(xr[HELD ? cc : 0], y[cc]) : zero;
                *reinterpret_cast<uint4 *>(dst) = hi;
                *reinterpret_cast<uint4 *>(D == 32 ? sOp + sw128_offset(r, 4 + pc) : dst + C::REST) = ok ? mul_rest_bf16x8(xr[HELD ? cc : 0], y[cc], hi) : zero;
            } else {
                *reinterpret_cast<uint4 *>(dst) = y[cc];
            }
        }
        return true;
    };
    constexpr int LPR = D / 8, RPI = 32 / LPR, LOADS = 32 / RPI;            // lanes per row, rows per load, loads of a warp
    const int brow = (warp & 3) * 32 + lane / LPR, bcc = lane % LPR;
    auto build_rows = [&](int t) -> bool {
        const int e = g.e0 + STEP * t + odd;
        const __nv_bfloat16 *bx = reinterpret_cast<const __nv_bfloat16 *>(tx.p) + elem_off(tx, b, 0, h) + bcc * 8, *by = ybase + bcc * 8;
        // loads [x0, x0 + m): operands of a row and, with SPLIT, what their product is not
        auto rows = [&](int x0, int m, uint4 *p, uint4 *rest) {
#pragma unroll
            for (int x = 0; x < m; ++x) {
                const int ii = g.i0 + ((brow + (x0 + x) * RPI) & (ROWS - 1)), kk = ii + kp.off2 - e;
                const bool ok = ii < kp.n && e < g.e1 && kk >= 0;
                p[x] = ok ? __ldg(reinterpret_cast<const uint4 *>(bx + (int64_t)ii * tx.sn)) : zero;
                rest[x] = ok ? __ldg(reinterpret_cast<const uint4 *>(by + (int64_t)kk * ty.sn)) : zero;
            }
#pragma unroll
            for (int x = 0; x < m; ++x) {
                const uint4 hi = mul_bf16x8(p[x], rest[x]);
                if constexpr (SPLIT) rest[x] = mul_rest_bf16x8(p[x], rest[x], hi);
                p[x] = hi;
            }
        };
        auto put = [&](int x0, int m, const uint4 *p, const uint4 *rest) {
#pragma unroll
            for (int x = 0; x < m; ++x) {
                const int row = brow + (x0 + x) * RPI;
                uint8_t *dst = sOp + (bcc >> 3) * C::BLK + sw128_offset(row, bcc & 7);
                *reinterpret_cast<uint4 *>(dst) = p[x];
                if constexpr (SPLIT) *reinterpret_cast<uint4 *>(D == 32 ? sOp + sw128_offset(row, 4 + bcc) : dst + C::REST) = rest[x];
            }
        };
        // the first products are formed before the wait for the stage, as many as there are registers for
        constexpr int FIRST = SPLIT ? 4 : 8, NEXT = 4;
        uint4 p[FIRST];
        {
            uint4 rest[4];
#pragma unroll
            for (int x = 0; x < FIRST; x += 4) rows(x, 4, p + x, rest);
            if (t >= 1 && !warp_wait(&bars[BQ_AB_EMPTY + WHICH], (t - 1) & 1, abort_flag, 3)) return false;
            put(0, FIRST, p, rest);
        }
#pragma unroll 1
        for (int x = FIRST; x < LOADS; x += NEXT) {
            uint4 q[NEXT], rest[NEXT];
            rows(x, NEXT, q, rest);
            put(x, NEXT, q, rest);
        }
        return true;
    };
    auto build = [&](int t) -> bool {
        bool done;
        if constexpr (HELD) done = build_held(t);
        else done = build_rows(t);
        if (!done) return false;
        fence_proxy_async_smem();
        mbar_arrive(&bars[BQ_AB_FULL + WHICH]);
        return true;
    };

    int slab_row = top_row, place = slab_row % C::RING;     // row of the slab and of the ring, of the next sweep
    auto drain = [&](int t) -> bool {
        bool ok;
        const uint4 *py = yrow(t, ok);
        auto xchunk = [&](int cc) { return __ldg(xrow + (cc ^ (rot / 8))); };
        auto ychunk = [&](int cc) { return ok ? __ldg(py + (cc ^ (rot / 8))) : zero; };
        if (!warp_wait(&bars[BQ_W_FULL + WHICH], t & 1, abort_flag, 1)) return false;
        tc_fence_after();
        // Up to head dim 64 half a row of U or W is read at a time, head dim 128 reads sixteen channels.
        constexpr int H = D / 2;
        uint32_t part[HELD ? H : 16];
        auto read = [&](int c) {
            if constexpr (D == 64) tmem_ld32(cols + (c ^ rot), part);
            else tmem_ld16(cols + (c ^ rot), part);
            tmem_wait_ld(part);
        };
        auto release = [&]() {            // the rest is in registers: the tensor cores may overwrite the accumulator
            tc_fence_before();
            mbar_arrive(&bars[BQ_W_EMPTY + WHICH]);
        };
        // every row of the ring belonged to other threads in the last sweep
        if (t >= 1 && !warp_wait(&bars[BQ_FOLD_SYNC + WHICH], (t - 1) & 1, abort_flag, 2)) return false;
        const bool sole = r == 63 || r == 64;           // (pairs) the first row of the sweep and the last have one writer
        const bool end = t == g.nsweeps - 1;
        float *row = acc + place * C::ACC_STRIDE;
        ulonglong2 *gone = reinterpret_cast<ulonglong2 *>(slab + (size_t)slab_row * D);
        // GROUP pieces of eight channels at a time: all their loads first, since every access to shared memory waits behind the
        // tensor cores' fetches (300 cycles and more)
        constexpr int GROUP = 2;
#pragma unroll
        for (int c0 = 0; c0 < NC; c0 += GROUP) {
            const bool second = c0 >= NC / 2;
            if (PAIR && c0 == NC / 2) {
                mbar_arrive(&bars[BQ_FOLD_MID + WHICH]);
                if (!warp_wait(&bars[BQ_FOLD_MID + WHICH], t & 1, abort_flag, 4)) return false;
            }
            // nothing has been added to the row (here: to these channels) yet / nothing will be after this
            const bool fresh = !PAIR ? t == 0 || r == 0 : second ? r == 64 || (t == 0 && r == 63) : t == 0 || r == 0 || r == 64 || r == 65;
            const bool out = !PAIR ? end || r == 127 : second ? end || r == 62 || r == 63 || r == 127 : r == 63 || (end && sole);
            uint4 xx[GROUP], yy[GROUP];
            ulonglong2 a[GROUP][2];
            auto place_of = [&](int g, int half) {          // first 16-byte piece of the eight floats, and the one behind it
                const int pc = 2 * ((c0 + g) ^ (rot / 8)) + half;
                return reinterpret_cast<ulonglong2 *>(row + 4 * (D == 128 ? pc ^ (place & 31) : pc));
            };
#pragma unroll
            for (int g = 0; g < GROUP; ++g) {
                xx[g] = yy[g] = zero;
                if constexpr (HELD) xx[g] = xr[HELD ? c0 + g : 0];
                else xx[g] = xchunk(c0 + g);
                if constexpr (STAGE_Y) yy[g] = ystaged(t, (c0 + g) ^ (rot / 8));
                else if constexpr (WHICH == 0) yy[g] = ychunk(c0 + g);
                a[g][0] = a[g][1] = make_ulonglong2(0, 0);
                if (!fresh) { a[g][0] = *place_of(g, 0); a[g][1] = *place_of(g, 1); }
            }
            if (!HELD || c0 % (NC / 2) == 0) {
                read(c0 * 8);
                if (HELD ? c0 == NC / 2 : c0 + GROUP == NC) release();
            }
#pragma unroll
            for (int g = 0; g < GROUP; ++g) {
                const int cc = c0 + g, pc = 2 * (cc ^ (rot / 8));
                const uint32_t xw[4] = {xx[g].x, xx[g].y, xx[g].z, xx[g].w}, yw[4] = {yy[g].x, yy[g].y, yy[g].z, yy[g].w};
                unsigned long long *const sum[4] = {&a[g][0].x, &a[g][0].y, &a[g][1].x, &a[g][1].y};
                if (ok) {
#pragma unroll
                    for (int z = 0; z < 4; ++z) {
                        const int q = (HELD ? cc * 8 % H : 8 * g) + 2 * z;
                        const uint64_t t2 = f2_pack(part[q], part[q + 1]);
                        if constexpr (WHICH == 0) dq[cc * 4 + z] = f2_fma(t2, f2_from_bf16x2(yw[z]), dq[cc * 4 + z]);
                        *sum[z] = f2_fma(t2, f2_from_bf16x2(xw[z]), *sum[z]);
                    }
                }
                if (out) {
                    gone[pc] = a[g][0];
                    gone[pc + 1] = a[g][1];
                } else {
                    *place_of(g, 0) = a[g][0];
                    *place_of(g, 1) = a[g][1];
                }
            }
        }
        mbar_arrive(&bars[BQ_FOLD_SYNC + WHICH]);
        slab_row -= STEP;
        place -= STEP;
        if (place < 0) place += C::RING;
        return true;
    };
    const int nv = g.total > 0 ? g.nsweeps : 0;       // a split whose units all lie before the sequence start has no work
    // (the first operands come from global memory: the tensor cores wait for them, and not for the staged copy)
    if (nv > 0 && !build(0)) return ERR_BQ_COMPUTE;
    if constexpr (STAGE_Y)
        if (nv > 0) stage();
    for (int t = 0; t < nv; ++t) {
        // the operands of the next sweep first: the tensor cores wait for them, U / W of this sweep arrive later
        if ((t + 1 < nv && !build(t + 1)) || !drain(t)) return ERR_BQ_COMPUTE;
    }
    return 0;
}

template <int D, bool SPLIT, bool PAIR, int WHICH>
__device__ __forceinline__ int bq_fold(const BqParams &P, const BqGeom &g, uint32_t tmem, float *acc, uint8_t *sOp, uint8_t *sStage, uint64_t *bars,
                                       volatile int *abort_flag) {
    const KernelParams &kp = P.kp;
    constexpr int ROWS = bq_rows(PAIR);
    const int r = threadIdx.x & 127, ir = r & (ROWS - 1), i = g.i0 + ir, rot = PAIR && r >> 6 ? D / 2 : 0;
    const int h = blockIdx.y, b = blockIdx.z;
    const int slab_rows = ROWS - 1 + P.epc;
    float *slab = P.part_k2 + (((((size_t)b * kp.hq + h) * P.nqt + g.qt) * P.nsplit + g.split) * 2 + WHICH) * (size_t)(slab_rows * D);
    uint64_t dq[WHICH ? 1 : D / 2];
    int err;
    if constexpr (WHICH == 0) err = bq_fold_body<D, SPLIT, PAIR, 0>(P, g, tmem, acc, sOp, sStage, slab, dq, bars, abort_flag);
    else {
        uint64_t none[D / 2];
        err = bq_fold_body<D, SPLIT, PAIR, 1>(P, g, tmem, acc, sOp, sStage, slab, none, bars, abort_flag);
    }
    const bool bad = err != 0 || *abort_flag != 0;     // a CTA in which a wait ran out reports NaN
    if constexpr (WHICH == 0) {
        // Pairs: the rows of the odd offsets hand their share of dQ over in shared memory: every product that reads A is done.
        float *buf = reinterpret_cast<float *>(sOp) + ir * D;
        auto piece = [&](int x) { return buf + 4 * (x ^ (ir & (D / 4 - 1))); };
        if (rot) {
#pragma unroll
            for (int x = 0; x < D / 4; ++x)
                *reinterpret_cast<ulonglong2 *>(piece(x ^ (D / 8))) = make_ulonglong2(dq[2 * x], dq[2 * x + 1]);
        }
        // (reached by a warp that gave up as well)
        if constexpr (PAIR) bq_fold_sync(0);
        if (!rot && i < kp.n) {
            // with one split per query tile dQ is final and goes straight to the gradient, otherwise a partial for the reduction
            float *dst = P.nsplit == 1 ? nullptr : P.part_dq + ((((size_t)g.split * kp.b + b) * kp.n + i) * kp.hq + h) * D;
            const int64_t o = elem_off(kp.dq, b, i, h);
#pragma unroll
            for (int x = 0; x < D / 4; ++x) {
                const float4 y = PAIR ? *reinterpret_cast<const float4 *>(piece(x)) : make_float4(0.f, 0.f, 0.f, 0.f);
                float v[4];
                f2_unpack(dq[2 * x], v[0], v[1]);
                f2_unpack(dq[2 * x + 1], v[2], v[3]);
                v[0] += y.x; v[1] += y.y; v[2] += y.z; v[3] += y.w;
#pragma unroll
                for (int z = 0; z < 4; ++z) v[z] = bad ? CUDART_NAN_F : dst ? v[z] : v[z] * kp.scale;
                if (dst) store_vec<4>(dst, 4 * x, false, v);
                else store_vec<4>(kp.dq.p, o + 4 * x, kp.grad_bf16 != 0, v);
            }
        }
    }
    if (bad)
        for (int x = r; x < slab_rows * D; x += 128) slab[x] = CUDART_NAN_F;
    return err;
}

template <int D, bool SPLIT, bool PAIR>
__global__ void __launch_bounds__(BqCfg<D, SPLIT, PAIR>::THREADS, 1)
bwd_q_kernel(const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapV, const BqParams P) {
    using C = BqCfg<D, SPLIT, PAIR>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = align_smem(smem_raw);
    uint8_t *sK = smem;
    uint8_t *sV = sK + C::KV_BYTES;
    uint8_t *sA = sV + C::KV_BYTES;
    uint8_t *sB = sA + C::TILE;
    float *acc_k = reinterpret_cast<float *>(sB + C::TILE), *acc_v = acc_k + C::ACC_BYTES / 4;
    uint8_t *sStage = reinterpret_cast<uint8_t *>(acc_v + C::ACC_BYTES / 4);
    uint64_t *bars = reinterpret_cast<uint64_t *>(sStage + C::STAGE_BYTES);
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bars + BQ_BAR_COUNT);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_holder + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);       // warp-uniform, and known to be
    if (threadIdx.x == 0) {
        for (int x = 0; x < BQ_BAR_COUNT; ++x) {
            const bool pfull = x >= BQ_P_FULL && x < BQ_P_FULL + 3;          // every compute thread
            const bool fold = (x >= BQ_W_EMPTY && x < BQ_W_EMPTY + 2) || (x >= BQ_FOLD_MID && x < BQ_FOLD_SYNC + 2) ||
                              (x >= BQ_AB_FULL && x < BQ_AB_FULL + 2);      // every thread of a fold group
            // S_FULL collects a commit from each of the two first-product issuers, G_DONE (up to head dim 64) from each of
            // the two second-product issuers
            const bool two = (x >= BQ_S_FULL && x < BQ_S_FULL + 3) || (D <= 64 && x >= BQ_G_DONE && x < BQ_G_DONE + 3);
            mbar_init(&bars[x], pfull ? 256u : fold ? 128u : two ? 2u : 1u);
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
    const BqGeom g = bq_geom<PAIR>(P, blockIdx.x / P.nsplit, blockIdx.x % P.nsplit);

    int err = 0;
#ifdef SA2_PROF
    const long long prof_t0 = clock64();
    sa2::sm100::prof_begin();
#endif
    if (warp < 4) {
        reg_dealloc<C::REGS_ISSUE>();                 // one instruction for the whole warpgroup
        if (g.total > 0) {
            if (warp == 0) err = bq_mma_second<D, SPLIT>(P, g, D <= 64 ? 0 : 2, &mapK, &mapV, tmem, sK, sV, bars, abort_flag);
            else if (warp == 1) err = bq_mma_first<D, SPLIT>(g, 0, tmem, sK, sA, bars, abort_flag);
            else if (warp == 2) err = bq_mma_first<D, SPLIT>(g, 1, tmem, sV, sB, bars, abort_flag);
            else if constexpr (D <= 64) err = bq_mma_second<D, SPLIT>(P, g, 1, &mapK, &mapV, tmem, sK, sV, bars, abort_flag);
            else err = bq_ring_producer<D, SPLIT>(P, g, &mapK, &mapV, sK, sV, bars, abort_flag);
        }
    } else if (warp < 12) {
        // one call site for both compute groups: they run the same instructions, which the instruction caches
        // of a scheduler then hold once (with two copies: 3.5 ms against 2.3)
        if constexpr (C::REGS_COMPUTE < C::REGS_LAUNCH) reg_dealloc<C::REGS_COMPUTE>();
        err = bq_compute<D, SPLIT, PAIR>(P, g, (warp >> 2) - 1, tmem, bars, abort_flag);
    } else if (warp < 16) {
        reg_alloc<C::REGS_FOLD>();
        err = bq_fold<D, SPLIT, PAIR, 0>(P, g, tmem, acc_k, sA, sStage, bars, abort_flag);
    } else {
        if constexpr (C::REGS_FOLD_W > C::REGS_LAUNCH) reg_alloc<C::REGS_FOLD_W>();
        err = bq_fold<D, SPLIT, PAIR, 1>(P, g, tmem, acc_v, sB, sStage, bars, abort_flag);
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

// ---------------------------------------------------------------------------
// Reduction of the partials: one thread per 4 channels of an output row.
//   dq[b,i,h]   = scale * sum_split part_dq[split][b][i][h]        (two or more splits only)
//   dk2[b,k,hk] = scale * sum_{h in group} sum_{tiles touching k} sum_split slab_k[...]
//   dv2[b,k,hk] =         same over slab_v
//   dk1[b,j,hk] = scale * sum_{split of the key tile} part_k1[...], dv1 the same (two or more splits only)
// Row k (position k - off2 in query coordinates) lies in the slab of query tile
// T of R rows and the split of offsets [e0, e0 + epc) at slab row k - off2 - R T + e0 + epc - 1, for the
// tiles where that index falls inside [0, R - 1 + epc) and among the rows of the sweeps that the CTA ran.
// ---------------------------------------------------------------------------
// GROUPED: more than one query head a key/value head and one split, four heads' loads at a time (with one head their registers would only
// cost blocks).  b2 n495 hq16 hk2 d32 w214/10 16.7 us with a head after the other -> 4.7.
template <int D, bool PAIR, bool GROUPED>
__global__ void __launch_bounds__(256) bwd_q_reduce_kernel(const BqParams P) {
    constexpr int TPR = D / 4;                          // threads per row
    constexpr int ROWS = bq_rows(PAIR);
    const KernelParams &kp = P.kp;
    const int acc_rows = ROWS - 1 + P.epc;
    const int64_t nq = !P.reduce_q || P.nsplit == 1 ? 0 : (int64_t)kp.b * kp.n * kp.hq * TPR;      // one split: dQ is already in place
    const int64_t nk = !P.reduce_q ? 0 : (int64_t)kp.b * kp.nk2 * kp.hk * TPR;
    const int64_t nk1 = !P.reduce_k1 ? 0 : (int64_t)kp.b * kp.nk1 * kp.hk * TPR;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool gbf16 = kp.grad_bf16 != 0;
    if (idx < nq) {
        const int c4 = (int)(idx % TPR) * 4;
        int64_t rest = idx / TPR;
        const int h = (int)(rest % kp.hq); rest /= kp.hq;
        const int i = (int)(rest % kp.n);
        const int b = (int)(rest / kp.n);
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s = 0; s < P.nsplit; ++s) {
            const float4 v = *reinterpret_cast<const float4 *>(P.part_dq + ((((size_t)s * kp.b + b) * kp.n + i) * kp.hq + h) * D + c4);
            acc[0] += v.x; acc[1] += v.y; acc[2] += v.z; acc[3] += v.w;
        }
#pragma unroll
        for (int z = 0; z < 4; ++z) acc[z] *= kp.scale;
        store_vec<4>(kp.dq.p, elem_off(kp.dq, b, i, h) + c4, gbf16, acc);
    } else if (idx < nq + nk) {
        const int64_t id2 = idx - nq;
        const int c4 = (int)(id2 % TPR) * 4;
        int64_t rest = id2 / TPR;
        const int hk = (int)(rest % kp.hk); rest /= kp.hk;
        const int k = (int)(rest % kp.nk2);
        const int b = (int)(rest / kp.nk2);
        float ak[4] = {0.f, 0.f, 0.f, 0.f}, av[4] = {0.f, 0.f, 0.f, 0.f};
        const int pos = k - kp.off2;                    // in query coordinates (may be negative for halo rows)
        // The slab rows of split s that hold row k: at most two tiles T with 0 <= pos - ROWS T + top < acc_rows, T1 and the one before it
        static_assert(ROWS - 1 + BQ_MAX_EPC <= 2 * ROWS, "two tiles at most");
        int T1, row[2];
        bool ok[2];
        auto find = [&](int s) {
            const int e0 = (s / P.tsplit) * P.epc, top = e0 + P.epc - 1;
            const int low = P.epc - (min(kp.w2 - e0, P.epc) + bq_step(PAIR) - 1) / bq_step(PAIR) * bq_step(PAIR);      // first row there is
            T1 = min(P.nqt - 1, pos + top >= 0 ? (pos + top) / ROWS : -1);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int T = T1 - 1 + x;
                row[x] = pos - ROWS * T + top;
                ok[x] = T >= 0 && row[x] >= low && row[x] < acc_rows;
                // (a tile that sees no start of the sequence has run all the split's sweeps, over units)
                if (ok[x] && (ROWS * T + kp.off2 < kp.w2 - 1 || ROWS * (T + 1) + kp.off1 < 64 * P.nu)) {
                    const BqGeom g = bq_geom<PAIR>(P, T, s);
                    ok[x] = g.nunits > 0 && row[x] >= P.epc - bq_step(PAIR) * g.nsweeps;
                }
            }
        };
        // all loads of a head before its sums: where they are not there a zero is added
        auto add = [&](int h, int s) {
            const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
            float4 vk[2], vv[2];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const float *slab = P.part_k2 + ((((size_t)b * kp.hq + h) * P.nqt + (T1 - 1 + x)) * P.nsplit + s) * (size_t)(2 * acc_rows * D) + c4;
                vk[x] = ok[x] ? *reinterpret_cast<const float4 *>(slab + (size_t)row[x] * D) : zero;
                vv[x] = ok[x] ? *reinterpret_cast<const float4 *>(slab + (size_t)(acc_rows + row[x]) * D) : zero;
            }
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                ak[0] += vk[x].x; ak[1] += vk[x].y; ak[2] += vk[x].z; ak[3] += vk[x].w;
                av[0] += vv[x].x; av[1] += vv[x].y; av[2] += vv[x].z; av[3] += vv[x].w;
            }
        };
        if constexpr (GROUPED) {
            find(0);
#pragma unroll 4
            for (int hh = 0; hh < kp.g; ++hh) add(hk * kp.g + hh, 0);
        } else {
#pragma unroll 1
            for (int hh = 0; hh < kp.g; ++hh)
#pragma unroll 1
                for (int s = 0; s < P.nsplit; ++s) {
                    find(s);
                    add(hk * kp.g + hh, s);
                }
        }
#pragma unroll
        for (int z = 0; z < 4; ++z) ak[z] *= kp.scale;
        store_vec<4>(kp.dk2.p, elem_off(kp.dk2, b, k, hk) + c4, gbf16, ak);
        store_vec<4>(kp.dv2.p, elem_off(kp.dv2, b, k, hk) + c4, gbf16, av);
    } else if (idx < nq + nk + nk1) {
        const int64_t id3 = idx - nq - nk, row = id3 / TPR, rows = (int64_t)kp.b * kp.nk1 * kp.hk;
        const int c4 = (int)(id3 % TPR) * 4;
        const int hk = (int)(row % kp.hk), j = (int)(row / kp.hk % kp.nk1), b = (int)(row / ((int64_t)kp.hk * kp.nk1));
        float ak[4] = {0.f, 0.f, 0.f, 0.f}, av[4] = {0.f, 0.f, 0.f, 0.f};
        for (int s = 0; s < P.ce; ++s) {
            const float *src = P.part_k1 + ((size_t)s * rows + row) * (2 * D) + c4;
            const float4 vk = *reinterpret_cast<const float4 *>(src), vv = *reinterpret_cast<const float4 *>(src + D);
            ak[0] += vk.x; ak[1] += vk.y; ak[2] += vk.z; ak[3] += vk.w;
            av[0] += vv.x; av[1] += vv.y; av[2] += vv.z; av[3] += vv.w;
        }
#pragma unroll
        for (int z = 0; z < 4; ++z) ak[z] *= kp.scale;
        store_vec<4>(kp.dk1.p, elem_off(kp.dk1, b, j, hk) + c4, gbf16, ak);
        store_vec<4>(kp.dv1.p, elem_off(kp.dv1, b, j, hk) + c4, gbf16, av);
    }
}

}  // namespace tc
}  // namespace sa2
