// Backward kernel for dQ, dK2, dV2 on tcgen05 tensor cores (bf16 operands,
// fp32 accumulation in TMEM, head dims 32, 64 and 128), plus the reduction of its
// partials and of those of dK1 / dV1.
//
// A CTA owns 128 query rows i of one (batch, query head) and a subset ("split")
// of the 128-row K1/V1 tiles of their window.  Because the backward recomputes
// probabilities from the saved logsumexp, the splits of one query tile are
// independent; each writes fp32 partials to scratch and a small second kernel
// adds them in a fixed order (splits, then the query heads of a kv group), so
// results are reproducible.
// Head dims 32 and 64: a split keeps its (at most three) tiles resident in shared memory; a 5-tile window is
// two splits; the offsets may be split as well (bq_split).
// Head dim 128: a CTA produces 64 of the 128 output channels (blockIdx.x also carries the channel
// half): S and dP contract over all 128 channels, U and W use the 64-channel block of K1 / V1 as their
// B operand, so the fold, its registers and the shared accumulators are those of head dim 64.  Shared
// memory cannot hold a window at this head dim, so one CTA walks the whole window (one split) and its
// 64-row units stream through a three-slot TMA ring (32 KB per slot), once per sweep, from L2: a slot is
// refilled when the U / W products of its unit are done, one unit ahead of the S / dP products that need it.
//
// SPLIT (head dim 32, and second windows above 56 rows: see bq_plan) keeps A_e, B_e, P and G as a bf16 value and a bf16 rest
// each, with twice the products; the rests cost a K1/V1 tile at head dim 64 and two of the three ring slots at 128.
//
// Per offset e ("sweep") the fold groups form A_e = q_i * k2_{i-e} and B_e = dO_i * v2_{i-e}; per 64-key
// unit the tensor cores compute
//     S = A_e K1^T      dP = B_e V1^T                 (rows i, columns j)
// the compute warps (one thread per query row and half of the unit's columns) form
//     P = exp2(c S - lse2_i)     G = P * (dP - D_i)    (bf16, back into TMEM)
// and the tensor cores accumulate over the sweep
//     U_e += G K1       W_e += P V1                    (K1/V1 as MN-major B)
// At the end of a sweep the row owner folds U_e, W_e into
//     dQ_i += U_e * k2_{i-e}                           (registers)
//     dK2_{i-e} += U_e * q_i,  dV2_{i-e} += W_e * dO_i (fp32 rows in shared memory)
// Row i-e of the shared accumulators is touched by exactly one thread per
// sweep, so the read-modify-write needs no atomics (see BqAcc for how the rows are kept).
//
// Warps: 0 issuer of U (up to head dim 64: after loading the tiles; head dim 128: of U and W); 1 TMEM owner and issuer of
// S; 2 issuer of dP; 3 issuer of W (head dim 128: TMA producer of the ring); 4-7 and 8-11 two compute groups, each
// forming 32 of the 64 columns of every unit (P, G).  Up to head dim 64 (640 threads) 12-15 form A_e of the next sweep
// and fold U of the last one into dQ / dK2, 16-19 do the same with B_e, W and dV2; at head dim 128 (512 threads) 12-15 do
// both (a second fold group and a third S / dP buffer there: 8.45 -> 9.2 ms on b1 n16384 h16 w512/32).
// TMEM columns: S / dP buffer x -> S/P [128x, 128x+64), dP/G [128x+64, 128x+128); P and G (bf16, 16 columns per
// 32 keys; at head dim 32 their rests in the next 16) overwrite the S and dP columns of the same keys - columns that the
// writing compute group has itself read - so a buffer is busy from the issue of S / dP until the U / W products of its unit are
// done.  Up to head dim 64 three such buffers are in flight (issue, compute and U / W of different units overlap) and
// there is one U / W accumulator pair [384, 512), which the fold groups read into registers before the next sweep's
// first product; head dim 128 has two buffers and U / W per sweep parity at [256 + 128p, +128).
//
// Bound, up to head dim 64: shared memory.  A unit's products fetch 512 cycles' worth of operands at 128 B/clk (S and dP:
// N = 64, so A is read again for every unit), the folds and the operand rows a further ~400, and everything that
// goes through shared memory - shuffles included - waits behind the tensor cores' fetches.  b4 n4096 h8 w512/32 takes
// ~1350 cycles a unit: 1.97 -> 1.58 ms at head dim 64, 40 -> 1.94 ms at 32 (the fp32 kernels before; 1.33 with A_e, B_e, P and
// G rounded to bf16: see bq_plan).  Measured and not
// kept: A_e and B_e in TMEM, double-buffered, which leaves two S / dP buffers (1.74 ms); k2 / v2 rows moved from lane to
// lane by shuffles instead of a row per lane from memory (1.70 ms).  Head dim 128 (two buffers, S and dP formed in
// both channel halves): 11.7 -> 8.5 ms on b1 n16384 h16; the chain S / dP -> P / G -> U / W of two buffers paces it.
#pragma once
#include "sa2_tc_bwd_k1.cuh"

namespace sa2 {
namespace tc {

// Register hand-over between warpgroups.  A group can only grow by what another has released, or its setmaxnreg
// never returns, so the budgets must add up to what the block was launched with.
//   head dim 128: four groups of 128; the fold group takes 232 (dQ, and the operands of the next sweep or a k2 row
//                 and chunks of U and W).
//   up to 64:     five groups of 96 (640 threads): the U fold takes 160 (dQ, q and k2 rows, 128 registers, and a
//                 chunk of U), the W fold 104.
template <int D, bool SPLIT> struct BqCfg {
    static constexpr bool TWO_FOLDS = D <= 64;                   // U and W have a fold group each
    static constexpr int THREADS = TWO_FOLDS ? 640 : 512;
    static constexpr int REGS_LAUNCH = TWO_FOLDS ? 96 : 128, REGS_ISSUE = 40, REGS_COMPUTE = TWO_FOLDS ? 88 : 120;
    static constexpr int REGS_FOLD = TWO_FOLDS ? 160 : 232, REGS_FOLD_W = TWO_FOLDS ? 104 : 0;
    static_assert(REGS_ISSUE + 2 * REGS_COMPUTE + REGS_FOLD + REGS_FOLD_W == THREADS / 128 * REGS_LAUNCH, "register pool must balance");
    static constexpr int CH = D == 128 ? 2 : 1;                  // channel halves = CTAs per (query tile, split)
    static constexpr int CC = D < 64 ? D : 64;                   // channels this CTA produces
    static constexpr int KSTEPS = D / 16;                        // K = 16 steps of S and dP
    static constexpr uint32_t BLK = TJ * 128;                    // A_e / B_e: one [128 rows][64 channels] swizzled block
    // SPLIT: A_e, B_e, P and G are each a bf16 value and a bf16 rest.  The rests of A_e / B_e fill the free half of the rows
    // at head dim 32 and take blocks of their own otherwise, for which K1 / V1 make room
    static constexpr uint32_t REST = D == 32 ? 64 : CH * BLK;    // bytes from an element of A_e / B_e to its rest
    static constexpr uint32_t TILE = CH * BLK * (SPLIT && D > 32 ? 2 : 1);        // A_e or B_e
    static constexpr int MAX_TILES = SPLIT && D == 64 ? 2 : 3;   // K1/V1 tiles of a split (head dims 32, 64)
    // K1 / V1 in shared memory: head dim 64 keeps three 128-row tiles of 16 KB resident; head dim 128 has a
    // ring of three 64-row units, each two [64 rows][64 channels] blocks of 8 KB
    static constexpr int NSLOT = SPLIT && D == 128 ? 1 : 3;
    static constexpr uint32_t KV_BYTES = D <= 64 ? MAX_TILES * BLK : NSLOT * 16384;
    static constexpr uint32_t UBLK = 8192;                       // one channel block of a 64-row unit (head dim 128)
    static constexpr int NBUF = D <= 64 ? 3 : 2;                 // S / dP (P / G) buffers in TMEM
    static constexpr int UWBUF = D <= 64 ? 1 : 2;                // U / W accumulator pairs in TMEM
    static constexpr uint32_t UW0 = NBUF * 128;                  // first TMEM column of U / W
};
// Shared accumulators of dK2 / dV2: in sweep e thread r adds to slab row r + epc - 1 - e (epc offsets per CTA), so 128 consecutive rows
// are live at a time.
// Head dims 32 and 64 keep all 127 + epc rows, 68 floats apart (64 + 4: the row-per-thread accesses of a warp spread over
// all banks, and the offsets inside a row are compile-time constants).
// Head dim 128 needs the space for its K1 / V1 ring and keeps a ring of 128 rows (slab row modulo 128): the top
// row of a sweep is complete when thread 127 has added to it; one warp copies it to the slab in global memory at
// the start of the next sweep, and thread 0 then writes (not adds to) the row that takes its place.  A row is 64
// floats; its sixteen 16-byte chunks are XOR-ed with the row number instead of padding.
constexpr int BQ_ACC_RING = 128;
constexpr int BQ_ACC_STRIDE = 68;
constexpr int BQ_MAX_EPC = 56;           // most offsets of a CTA: 127 + epc accumulator rows must fit (head dim 64)
template <int D> struct BqAcc {
    static constexpr bool RING = D == 128;
    __host__ __device__ static int rows(int epc) { return RING ? BQ_ACC_RING : 127 + epc; }
    __host__ __device__ static int row_floats() { return RING ? 64 : BQ_ACC_STRIDE; }
    // float index of (slab row, channel col) inside one accumulator array, col % 4 == 0
    __device__ static int off(int slab_row, int col) {
        if constexpr (RING) {
            const int pr = slab_row & (BQ_ACC_RING - 1);
            return pr * 64 + ((((col >> 2) ^ pr) & 15) << 2);
        } else {
            return slab_row * BQ_ACC_STRIDE + col;
        }
    }
};

// With a fold group each for U and W (head dims 32 and 64), entry 0 of a pair belongs to A_e, S, U and entry 1 to B_e,
// dP, W, except S_FULL ... G_DONE; at head dim 128 A and B share entry 0, and U and W share the entry of their parity.
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
    BQ_FOLD_SYNC = 24,   // [2] every fold thread has added its sweep into the shared accumulators
    BQ_BAR_COUNT = 26
};

enum { ERR_BQ_PRODUCER = 256, ERR_BQ_MMA = 512, ERR_BQ_COMPUTE = 1024, ERR_BQ_BUILDER = 2048 };

struct BqParams {
    KernelParams kp;
    float c;            // scale * log2(e)
    int nt;             // K1/V1 tiles per query tile
    int nsplit;         // CTAs sharing one query tile: tsplit x (offset splits)
    int tsplit;         // splits of the K1/V1 window
    int tiles_per_split;
    int epc;            // second-key offsets of a CTA: split s takes [epc * (s / tsplit), +epc)
    int nqt;            // query tiles
    float *part_dq;     // [nsplit][b][n][hq][d]
    float *part_k2;     // [b][hq][nqt][nsplit][2][127 + epc][d]   (dK2 slab, then dV2 slab)
    int *status;
    // what the reduction adds up: dQ and dK2/dV2, and the dK1/dV1 partials of ce CTAs per key tile
    const float *part_k1;
    int ce, reduce_q, reduce_k1;
};

template <int D, bool SPLIT> inline size_t bq_smem_bytes(int epc) {
    return 1024 + (size_t)2 * BqCfg<D, SPLIT>::KV_BYTES + 2 * BqCfg<D, SPLIT>::TILE +
           (size_t)2 * BqAcc<D>::rows(epc) * BqAcc<D>::row_floats() * sizeof(float) + 256;
}
// (a query tile with one split writes dQ itself and needs no partials)
inline size_t bq_part_dq_bytes(const sa2_shape &s, int nsplit) { return nsplit == 1 ? 0 : (size_t)nsplit * s.b * s.n * s.hq * s.d * sizeof(float); }
inline size_t bq_part_k2_bytes(const sa2_shape &s, int nsplit, int epc) {
    const size_t nqt = (s.n + TQ - 1) / TQ;
    return (size_t)s.b * s.hq * nqt * nsplit * 2 * (127 + epc) * s.d * sizeof(float);
}

struct BqGeom {
    int qt, split, chh;          // query tile, split, channel half of this CTA
    int i0, i_last, nsweeps;
    int e0;                      // first offset of the CTA: sweep e is offset e0 + e
    int ubase;                   // first-key row of the CTA's unit 0; unit x covers rows ubase + 64 x ... + 63
    int nunits;                  // 64-key units the CTA visits in every sweep
    int total;                   // nunits * nsweeps
};

template <int D>
__device__ __forceinline__ BqGeom bq_geom(const BqParams &P) {
    BqGeom g;
    const KernelParams &kp = P.kp;
    constexpr int CH = D == 128 ? 2 : 1;
    g.chh = blockIdx.x % CH;
    const int qs = blockIdx.x / CH;
    g.qt = qs / P.nsplit;
    g.split = qs % P.nsplit;
    g.i0 = g.qt * TQ;
    g.i_last = min(g.i0 + TQ - 1, kp.n - 1);
    g.e0 = (g.split / P.tsplit) * P.epc;
    g.nsweeps = max(0, min(min(kp.w2, g.e0 + P.epc), g.i_last + kp.off2 + 1) - g.e0);
    const int ts = g.split % P.tsplit;
    if constexpr (D <= 64) {
        const int jbase = g.i0 + kp.off1 + TJ - TJ * P.nt;        // tile t covers rows jbase + 128 t ...
        const int t_first = jbase >= 0 ? 0 : min(P.nt - 1, (-jbase) / TJ);
        const int t_begin = max(t_first, ts * P.tiles_per_split);
        const int t_end = min(P.nt, (ts + 1) * P.tiles_per_split);
        g.ubase = jbase + TJ * t_begin;
        g.nunits = 2 * max(0, t_end - t_begin);
    } else {
        const int nh = (kp.w1 + TQ - 1 + 63) / 64;                // 64-row units of the window: ceil((w1 + 127) / 64)
        const int hbase = g.i0 + kp.off1 + TQ - 64 * nh;
        const int h_first = hbase >= 0 ? 0 : min(nh - 1, (-hbase) / 64);
        g.ubase = hbase + 64 * h_first;
        g.nunits = nh - h_first;
    }
    g.total = g.nunits * g.nsweeps;
    return g;
}

// ---------------------------------------------------------------- issuers of S (warp 1) and dP (warp 2)
// Unit u (numbered over the whole kernel) is unit u % nunits of sweep u / nunits and uses TMEM buffer u % NBUF.
// A warp issues about one tcgen05.mma per 45-90 cycles, so the two product stages have an issuing warp
// each; U / W are accumulated by one warp only, which keeps the summation order fixed.
// which = 0: S = A_e K1^T into columns [128 buf, +64); which = 1: dP = B_e V1^T into [128 buf + 64, +64).
template <int D, bool SPLIT>
__device__ __forceinline__ int bq_mma_first(const BqGeom &g, int which, uint32_t tmem, uint8_t *sKV, uint8_t *sAB,
                                            uint64_t *bars, volatile int *abort_flag) {
    using C = BqCfg<D, SPLIT>;
    constexpr uint32_t IDESC_F = idesc_bf16(128, 64, false, false);
    const uint64_t dT = smem_desc_sw128(smem_u32(sKV)), dA = smem_desc_sw128(smem_u32(sAB));
    if constexpr (D <= 64) {
        if (!mbar_wait_warp(&bars[BQ_KV_FULL], 0, abort_flag)) return ERR_BQ_MMA;
    }
    const int ab = C::TWO_FOLDS ? which : 0;
    int u = 0, buf = 0, use = 0;                         // use = u / NBUF: how often the buffer has been used before
    int slot = 0, suse = 0;                              // head dim 128: ring slot u % NSLOT and u / NSLOT
    for (int e = 0; e < g.nsweeps; ++e) {
        if (!mbar_wait_warp(&bars[BQ_AB_FULL + ab], e & 1, abort_flag, 0, 1)) return ERR_BQ_MMA;
        for (int w = 0; w < g.nunits; ++w, ++u) {
            // the buffer holds P / G of its previous unit until the U / W products of that unit are done
            if (use >= 1 && !mbar_wait_warp(&bars[BQ_G_DONE + buf], (use - 1) & 1, abort_flag, 0, 2)) return ERR_BQ_MMA;
            if constexpr (D == 128) {
                if (!mbar_wait_warp(&bars[BQ_KV_SLOT + slot], suse & 1, abort_flag, 0, 3)) return ERR_BQ_MMA;
            }
            tc_fence_after();
            SA2_PROF_MARK(seg);
            if (elect_one()) {
            const uint32_t d = tmem + buf * 128 + which * 64;
            if constexpr (D <= 64) {
                const uint64_t t = dT + (uint64_t)((w * 8192) >> 4);       // unit w: rows [64 w, +64) of the resident tiles
#pragma unroll
                for (int k = 0; k < C::KSTEPS; ++k) mma_ss(d, dA + 2 * k, t + 2 * k, IDESC_F, k > 0 ? 1u : 0u);
                if constexpr (SPLIT) {
#pragma unroll
                    for (int k = 0; k < C::KSTEPS; ++k) mma_ss(d, dA + (C::REST >> 4) + 2 * k, t + 2 * k, IDESC_F, 1u);
                }
            } else {
                const uint64_t t = dT + (uint64_t)((slot * 2 * C::UBLK) >> 4);
#pragma unroll
                for (int k = 0; k < (SPLIT ? 16 : 8); ++k)
                    mma_ss(d, dA + (uint64_t)(((k >> 2) * C::BLK) >> 4) + (uint64_t)((k & 3) * 2),
                           t + (uint64_t)(((k >> 2 & 1) * C::UBLK) >> 4) + (uint64_t)((k & 3) * 2), IDESC_F, k > 0 ? 1u : 0u);
            }
            SA2_PROF_LAP(4, seg);                         // issue of the products
            tc_commit(&bars[BQ_S_FULL + buf]);
            SA2_PROF_LAP(5, seg);                         // the commit
            }
            if (++buf == C::NBUF) { buf = 0; ++use; }
            if (++slot == C::NSLOT) { slot = 0; ++suse; }
        }
        if (elect_one()) tc_commit(&bars[BQ_AB_EMPTY + ab]);
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
// part 0 (warp 0; head dim 64: after loading the tiles): U += G K1; part 1 (warp 3): W += P V1; part 2 (head dim
// 128, warp 0): both.  Each accumulator has one issuing warp, which keeps its summation order fixed.
template <int D, bool SPLIT>
__device__ __forceinline__ int bq_mma_second(const BqParams &P, const BqGeom &g, int part, const CUtensorMap *mapK, const CUtensorMap *mapV,
                                             uint32_t tmem, uint8_t *sK, uint8_t *sV, uint64_t *bars, volatile int *abort_flag) {
    using C = BqCfg<D, SPLIT>;
    constexpr uint32_t IDESC_G = idesc_bf16(128, C::CC, false, true);
    if constexpr (D <= 64) {
        if (part == 0) {
            const int hk = blockIdx.y / P.kp.g;
            prefetch_tmap(mapK);
            prefetch_tmap(mapV);
            const int nt = g.nunits / 2;
            if (elect_one()) {
            mbar_arrive_expect_tx(&bars[BQ_KV_FULL], 2 * C::BLK * nt);
            for (int t = 0; t < nt; ++t) {
                const int row = g.ubase + TJ * t;
                tma_load_4d(sK + (size_t)t * C::BLK, mapK, &bars[BQ_KV_FULL], 0, hk, row, blockIdx.z);
                tma_load_4d(sV + (size_t)t * C::BLK, mapV, &bars[BQ_KV_FULL], 0, hk, row, blockIdx.z);
            }
            }
        }
        if (!mbar_wait_warp(&bars[BQ_KV_FULL], 0, abort_flag)) return ERR_BQ_PRODUCER;
    }
    // head dim 128: U / W take the CTA's 64-channel block of the unit as an MN-major B operand
    const uint64_t dK = smem_desc_sw128(smem_u32(sK) + (D <= 64 ? 0 : g.chh * C::UBLK));
    const uint64_t dV = smem_desc_sw128(smem_u32(sV) + (D <= 64 ? 0 : g.chh * C::UBLK));
    int u = 0, buf = 0, use = 0, slot = 0;
    for (int e = 0; e < g.nsweeps; ++e) {
        const int wb = e % C::UWBUF, wuse = e / C::UWBUF;
        const int wbar = C::TWO_FOLDS ? part : wb;
        const uint32_t tu = tmem + C::UW0 + wb * 128, tw = tu + 64;
        for (int w = 0; w < g.nunits; ++w, ++u) {
            if (!mbar_wait_warp(&bars[BQ_P_FULL + buf], use & 1, abort_flag, 0, 1)) return ERR_BQ_MMA;
            // the fold group must have read the accumulators of the sweep that used them last
            if (w == 0 && wuse >= 1 && !mbar_wait_warp(&bars[BQ_W_EMPTY + wbar], (wuse - 1) & 1, abort_flag, 0, 2)) return ERR_BQ_MMA;
            tc_fence_after();
            const uint64_t off = (uint64_t)((D <= 64 ? w * 8192 : slot * 2 * C::UBLK) >> 4);
            const uint64_t kt = dK + off, vt = dV + off;
            const uint32_t a = tmem + buf * 128;
            const uint32_t acc = w > 0 ? 1u : 0u;
            if (elect_one()) {
            if (part != 1) {
                // keys [32 x, +32) of G are 16 columns at 64 + 32 x, those of P at 32 x
                mma_ts(tu, a + 64, kt, IDESC_G, acc);               // U += G K1
                mma_ts(tu, a + 72, kt + 128, IDESC_G, 1u);
                mma_ts(tu, a + 96, kt + 256, IDESC_G, 1u);
                mma_ts(tu, a + 104, kt + 384, IDESC_G, 1u);
                if constexpr (SPLIT) {                              // the rests of G, behind it
                    mma_ts(tu, a + 80, kt, IDESC_G, 1u);
                    mma_ts(tu, a + 88, kt + 128, IDESC_G, 1u);
                    mma_ts(tu, a + 112, kt + 256, IDESC_G, 1u);
                    mma_ts(tu, a + 120, kt + 384, IDESC_G, 1u);
                }
            }
            if (part != 0) {
                mma_ts(tw, a, vt, IDESC_G, acc);                    // W += P V1
                mma_ts(tw, a + 8, vt + 128, IDESC_G, 1u);
                mma_ts(tw, a + 32, vt + 256, IDESC_G, 1u);
                mma_ts(tw, a + 40, vt + 384, IDESC_G, 1u);
                if constexpr (SPLIT) {
                    mma_ts(tw, a + 16, vt, IDESC_G, 1u);
                    mma_ts(tw, a + 24, vt + 128, IDESC_G, 1u);
                    mma_ts(tw, a + 48, vt + 256, IDESC_G, 1u);
                    mma_ts(tw, a + 56, vt + 384, IDESC_G, 1u);
                }
            }
            tc_commit(&bars[BQ_G_DONE + buf]);
            if constexpr (D == 128) tc_commit(&bars[BQ_KV_FREE + slot]);
            }
            if (++buf == C::NBUF) { buf = 0; ++use; }
            if (++slot == C::NSLOT) slot = 0;
        }
        if (elect_one()) tc_commit(&bars[BQ_W_FULL + wbar]);
    }
    return 0;
}

// ---------------------------------------------------------------- compute (warps 4-7; head dim 64: and 8-11): P and G
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
// Head dim 64: group cg forms columns [32 cg, +32) of every unit, which halves the time between S / dP and P / G.
template <int D, bool SPLIT>
__device__ __forceinline__ int bq_compute(const BqParams &P, const BqGeom &g, int cg, uint32_t tmem, uint64_t *bars, volatile int *abort_flag) {
    using C = BqCfg<D, SPLIT>;
    const KernelParams &kp = P.kp;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = (warp & 3) * 32 + lane;             // query row within the tile = TMEM lane
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int h = blockIdx.y, b = blockIdx.z;
    const int i = g.i0 + r;
    const bool row_ok = i < kp.n;
    const float c = P.c;
    float lse2 = 0.f, dl = 0.f;
    if (row_ok) {
        const int64_t o = ((int64_t)b * kp.hq + h) * kp.n + i;
        lse2 = kp.lse[o] * 1.4426950408889634f;
        dl = kp.delta[o];
    }
    const uint64_t c2 = f2_pack(c, c), nlse2 = f2_pack(-lse2, -lse2), ndl2 = f2_pack(-dl, -dl);
#ifdef SA2_PROF
    long long seg_ld = 0, seg_math = 0, seg_st = 0;       // cycles in TMEM loads, arithmetic, TMEM stores and hand-over
#endif
    {
        int e = 0, w = 0;
        for (int u = 0; u < g.total; ++u, ++w) {
            if (w == g.nunits) { w = 0; ++e; }
            const bool sweep_ok = row_ok && (i + kp.off2 - g.e0 - e >= 0);
            {
                const int buf = u % C::NBUF, use = u / C::NBUF;
                const int j0 = g.ubase + 64 * w;
                const int d1 = i + kp.off1 - j0;
                const int hi = sweep_ok ? min(d1, 63) : -1;         // valid columns: lo < col <= hi
                const int lo = max(d1 - kp.w1, -j0 - 1);
                if (!warp_wait(&bars[BQ_S_FULL + buf], use & 1, abort_flag, 1)) return ERR_BQ_COMPUTE;
                tc_fence_after();
                const bool full = __all_sync(0xffffffffu, lo < 0 && hi >= 63);
                {
                    const int ch = cg;
                    uint32_t sv[32], dv[32], pp[16], gg[16], pr[SPLIT ? 16 : 1], gr[SPLIT ? 16 : 1];
                    // no row of this warp has a valid column among these 32: P = G = 0 without reading S / dP
                    if (__all_sync(0xffffffffu, hi < ch * 32 || lo >= ch * 32 + 31)) {
#pragma unroll
                        for (int x = 0; x < 16; ++x) { pp[x] = 0u; gg[x] = 0u; pr[SPLIT ? x : 0] = 0u; gr[SPLIT ? x : 0] = 0u; }
                    } else {
#ifdef SA2_PROF
                    const long long seg_t0 = clock64();
#endif
                    tmem_ld32(lane_addr + buf * 128 + ch * 32, sv);
                    tmem_ld32(lane_addr + buf * 128 + 64 + ch * 32, dv);
                    tmem_wait_ld();
#ifdef SA2_PROF
                    const long long seg_t1 = clock64();
                    seg_ld += seg_t1 - seg_t0;
#endif
                    auto pg = [&](int x, float a0, float a1) {
                        pg_pair<SPLIT>(ex2(a0), ex2(a1), dv[x], dv[x + 1], ndl2, pp[x >> 1], gg[x >> 1], pr[SPLIT ? x >> 1 : 0], gr[SPLIT ? x >> 1 : 0]);
                    };
                    if (full) {
#pragma unroll
                        for (int x = 0; x < 32; x += 2) {
                            float a0, a1;
                            f2_unpack(f2_fma(f2_pack(sv[x], sv[x + 1]), c2, nlse2), a0, a1);
                            pg(x, a0, a1);
                        }
                    } else {
                        // valid columns are the integers in (lo, hi]: 2048 (half + 1/2 - |col - mid|) is at least 1024
                        // inside and at most -1024 outside, so the minimum with it leaves the exponents of valid cells
                        // alone and makes P exactly 0 elsewhere, whatever S is there (FMA pipe instead of compares and
                        // selects on the ALU pipe; all values are exact)
                        const float mid = 1024.f * (float)(lo + 1 + hi) - 2048.f * (float)(ch * 32), half = 1024.f * (float)(hi - lo);
#pragma unroll
                        for (int x = 0; x < 32; x += 2) {
                            float a0, a1;
                            f2_unpack(f2_fma(f2_pack(sv[x], sv[x + 1]), c2, nlse2), a0, a1);
                            a0 = fminf(a0, half - fabsf(2048.f * x - mid));
                            a1 = fminf(a1, half - fabsf(2048.f * (x + 1) - mid));
                            pg(x, a0, a1);
                        }
                    }
#ifdef SA2_PROF
                    seg_math += clock64() - seg_t1;
#endif
                    }
                    // P / G chunk over the first half of the columns of S / dP that this thread has just read (the
                    // other columns of the buffer may still be unread by the other compute group)
                    tmem_st16(lane_addr + buf * 128 + ch * 32, pp);
                    tmem_st16(lane_addr + buf * 128 + 64 + ch * 32, gg);
                    if constexpr (SPLIT) {
                        tmem_st16(lane_addr + buf * 128 + ch * 32 + 16, pr);
                        tmem_st16(lane_addr + buf * 128 + 64 + ch * 32 + 16, gr);
                    }
                }
#ifdef SA2_PROF
                const long long seg_t2 = clock64();
#endif
                tmem_wait_st();
                tc_fence_before();
                mbar_arrive(&bars[BQ_P_FULL + buf]);
#ifdef SA2_PROF
                seg_st += clock64() - seg_t2;
#endif
            }
        }
    }
    SA2_PROF_ADD(4, seg_ld);
    SA2_PROF_ADD(5, seg_math);
    SA2_PROF_ADD(6, seg_st);
    return 0;
}

// ---------------------------------------------------------------- fold: U, W -> dQ, dK2, dV2
// (which: the fold group of U, or of both; 1: that of W)
__device__ __forceinline__ void bq_fold_sync(int which) { asm volatile("bar.sync %0, 128;" ::"r"(1 + which) : "memory"); }

// dQ of one row (NaN when a wait ran out, so that the failure is visible in the result): with one split per query tile
// it is final and goes straight to the gradient, otherwise a partial for the reduction kernel
template <int D, int N>
__device__ __forceinline__ void bq_store_dq(const BqParams &P, const BqGeom &g, int i, const uint64_t (&dq2)[N], bool bad) {
    const KernelParams &kp = P.kp;
    const int h = blockIdx.y, b = blockIdx.z, c0 = g.chh * 64;
    float dq[2 * N];
#pragma unroll
    for (int x = 0; x < N; ++x) f2_unpack(dq2[x], dq[2 * x], dq[2 * x + 1]);
    if (P.nsplit == 1) {
        const bool gbf16 = kp.grad_bf16 != 0;
        const int64_t o = elem_off(kp.dq, b, i, h) + c0;
#pragma unroll
        for (int x = 0; x < 2 * N; x += 4) {
            float v[4];
#pragma unroll
            for (int z = 0; z < 4; ++z) v[z] = bad ? CUDART_NAN_F : dq[x + z] * kp.scale;
            store_vec<4>(kp.dq.p, o + x, gbf16, v);
        }
    } else {
        float *dst = P.part_dq + ((((size_t)g.split * kp.b + b) * kp.n + i) * kp.hq + h) * D + c0;
#pragma unroll
        for (int x = 0; x < 2 * N; x += 4)
            *reinterpret_cast<float4 *>(dst + x) = bad ? make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F)
                                                       : make_float4(dq[x], dq[x + 1], dq[x + 2], dq[x + 3]);
    }
}

__device__ __forceinline__ uint4 mul_bf16x8(const uint4 &x, const uint4 &y) {
    return make_uint4(mul_bf16x2(x.x, y.x), mul_bf16x2(x.y, y.y), mul_bf16x2(x.z, y.z), mul_bf16x2(x.w, y.w));
}

// Head dims 32 and 64: WHICH = 0 forms A_e = q_i * k2_{i-e} and folds U_e into dQ_i (registers) and dK2_{i-e};
// WHICH = 1 forms B_e = dO_i * v2_{i-e} and folds W_e into dV2_{i-e}.  One thread per query row; its q (dO) row stays
// in its registers.  With one group for both, U / W of the next sweep waited ~1960 of 9400 cycles a sweep for the
// accumulators to be read and S / dP ~1000 for their operands.
template <int D, bool SPLIT, int WHICH>
__device__ __forceinline__ int bq_fold_half(const BqParams &P, const BqGeom &g, uint32_t tmem, float *acc, uint8_t *sOp, uint64_t *bars,
                                            volatile int *abort_flag) {
    using C = BqCfg<D, SPLIT>;
    const KernelParams &kp = P.kp;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = (warp & 3) * 32 + lane;             // query row within the tile = TMEM lane
    const uint32_t cols = tmem + ((uint32_t)((warp & 3) * 32) << 16) + C::UW0 + WHICH * 64;
    const int h = blockIdx.y, b = blockIdx.z, hk = h / kp.g;
    const int i = g.i0 + r;
    const bool row_ok = i < kp.n;
    constexpr int NC = D / 8;                         // 16-byte chunks of a row
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const TensorRef &tx = WHICH ? kp.dout : kp.q, &ty = WHICH ? kp.v2 : kp.k2;
    uint4 xr[NC];
    {
        const uint4 *px = reinterpret_cast<const uint4 *>(reinterpret_cast<const __nv_bfloat16 *>(tx.p) + elem_off(tx, b, row_ok ? i : 0, h));
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) xr[cc] = row_ok ? __ldg(px + cc) : zero;
    }
    const __nv_bfloat16 *ybase = reinterpret_cast<const __nv_bfloat16 *>(ty.p) + elem_off(ty, b, 0, hk);
    uint64_t dq[WHICH ? 2 : D / 2];                   // pairs of channels
#pragma unroll
    for (int x = 0; x < (WHICH ? 2 : D / 2); ++x) dq[x] = 0;
#ifdef SA2_PROF
    long long seg_build = 0, seg_drain = 0;           // cycles after the waits of a build and of a fold
#endif
    auto yrow = [&](int e, bool &ok) {
        const int kk = i + kp.off2 - g.e0 - e;
        ok = row_ok && kk >= 0;
        return reinterpret_cast<const uint4 *>(ybase + (int64_t)(ok ? kk : 0) * ty.sn);
    };
    auto build = [&](int e) -> bool {
        bool ok;
        const uint4 *py = yrow(e, ok);
        uint4 y[NC];
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) y[cc] = ok ? __ldg(py + cc) : zero;
        if constexpr (!SPLIT) {
#pragma unroll
            for (int cc = 0; cc < NC; ++cc) y[cc] = ok ? mul_bf16x8(xr[cc], y[cc]) : zero;
        }
        if (e >= 1 && !warp_wait(&bars[BQ_AB_EMPTY + WHICH], (e - 1) & 1, abort_flag, 3)) return false;
#ifdef SA2_PROF
        const long long seg_t0 = clock64();
#endif
#pragma unroll
        for (int cc = 0; cc < NC; ++cc) {
            uint8_t *dst = sOp + sw128_offset(r, cc);
            if constexpr (SPLIT) {       // (formed here: a row of products and one of rests would not fit the registers)
                const uint4 hi = ok ? mul_bf16x8(xr[cc], y[cc]) : zero;
                *reinterpret_cast<uint4 *>(dst) = hi;
                *reinterpret_cast<uint4 *>(D == 32 ? sOp + sw128_offset(r, 4 + cc) : dst + C::REST) = ok ? mul_rest_bf16x8(xr[cc], y[cc], hi) : zero;
            } else {
                *reinterpret_cast<uint4 *>(dst) = y[cc];
            }
        }
        fence_proxy_async_smem();
        mbar_arrive(&bars[BQ_AB_FULL + WHICH]);
#ifdef SA2_PROF
        seg_build += clock64() - seg_t0;
#endif
        return true;
    };
    auto drain = [&](int e) -> bool {
        bool ok;
        const uint4 *py = yrow(e, ok);
        // The k2 row is fetched before the wait: shared memory leaves 28 KB of L1, so it often comes from L2 (with the
        // chunks fetched one step ahead of their use: 1.60 against 1.58 ms on b4 n4096 h8, head dim 64).
        uint4 yd[WHICH ? 1 : NC];
        if constexpr (WHICH == 0) {
#pragma unroll
            for (int cc = 0; cc < NC; ++cc) yd[cc] = ok ? __ldg(py + cc) : zero;
        }
        if (!warp_wait(&bars[BQ_W_FULL + WHICH], e & 1, abort_flag, 1)) return false;
        // A row of the shared accumulator is written by thread r in this sweep and by another thread in the
        // last one: every fold thread must have finished that one first.
        if (e >= 1 && !warp_wait(&bars[BQ_FOLD_SYNC + WHICH], (e - 1) & 1, abort_flag, 2)) return false;
        tc_fence_after();
#ifdef SA2_PROF
        const long long seg_t0 = clock64();
#endif
        float *arow = acc + (size_t)(r + P.epc - 1 - e) * BQ_ACC_STRIDE;
        constexpr int CH = 16;                        // channels per TMEM read
#pragma unroll
        for (int c = 0; c < D; c += CH) {
            uint32_t t[CH];
            tmem_ld16(cols + c, t);
            tmem_wait_ld();
            if (c + CH == D) {
                // the rest is in registers: the tensor cores may overwrite the accumulator
                tc_fence_before();
                mbar_arrive(&bars[BQ_W_EMPTY + WHICH]);
            }
            if (ok) {
#pragma unroll
                for (int p = 0; p < 2; ++p) {
                    const int ch = c + 8 * p;
                    const uint4 yy = yd[WHICH ? 0 : ch / 8];
                    const uint32_t xw[4] = {xr[ch / 8].x, xr[ch / 8].y, xr[ch / 8].z, xr[ch / 8].w}, yw[4] = {yy.x, yy.y, yy.z, yy.w};
                    ulonglong2 *dst = reinterpret_cast<ulonglong2 *>(arow + ch);
                    ulonglong2 a[2] = {dst[0], dst[1]};
                    unsigned long long *const sum[4] = {&a[0].x, &a[0].y, &a[1].x, &a[1].y};
#pragma unroll
                    for (int z = 0; z < 4; ++z) {
                        const uint64_t t2 = f2_pack(t[8 * p + 2 * z], t[8 * p + 2 * z + 1]);
                        if constexpr (WHICH == 0) dq[ch / 2 + z] = f2_fma(t2, f2_from_bf16x2(yw[z]), dq[ch / 2 + z]);
                        *sum[z] = f2_fma(t2, f2_from_bf16x2(xw[z]), *sum[z]);
                    }
                    dst[0] = a[0];
                    dst[1] = a[1];
                }
            }
        }
        mbar_arrive(&bars[BQ_FOLD_SYNC + WHICH]);
#ifdef SA2_PROF
        seg_drain += clock64() - seg_t0;
#endif
        return true;
    };
    const int nv = g.total > 0 ? g.nsweeps : 0;       // a split whose tiles all lie before the sequence start has no work
    int err = 0;
    if (nv > 0 && !build(0)) err = ERR_BQ_COMPUTE;
    for (int e = 0; e < nv && err == 0; ++e) {
        // the operands of the next sweep first: the tensor cores wait for them, U / W of this sweep arrive later
        if ((e + 1 < nv && !build(e + 1)) || !drain(e)) err = ERR_BQ_COMPUTE;
    }
    SA2_PROF_ADD(4, seg_build);
    SA2_PROF_ADD(5, seg_drain);
    if constexpr (WHICH == 0) {
        if (row_ok) bq_store_dq<D>(P, g, i, dq, err != 0 || *abort_flag != 0);
    }
    return err;
}

// Head dim 128: one group for both.

template <int D, bool SPLIT>
__device__ __forceinline__ int bq_fold_body(const BqParams &P, const BqGeom &g, uint32_t tmem, float *acc_k, float *acc_v, float *slab,
                                            uint8_t *sA, uint8_t *sB, uint64_t *bars, volatile int *abort_flag) {
    using C = BqCfg<D, SPLIT>;
    const KernelParams &kp = P.kp;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r = (warp & 3) * 32 + lane;             // query row within the tile = TMEM lane
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const int h = blockIdx.y, b = blockIdx.z, hk = h / kp.g;
    const int c0 = g.chh * 64;                        // first channel this CTA produces
    const int i = g.i0 + r;
    const bool row_ok = i < kp.n;
    constexpr int NC = C::CC / 8;                     // 16-byte chunks of the CTA's channels
    uint64_t dq[C::CC / 2];                           // pairs of channels
#pragma unroll
    for (int x = 0; x < C::CC / 2; ++x) dq[x] = 0;
    const __nv_bfloat16 *qrow = reinterpret_cast<const __nv_bfloat16 *>(kp.q.p) + elem_off(kp.q, b, row_ok ? i : 0, h) + c0;
    const __nv_bfloat16 *dorow = reinterpret_cast<const __nv_bfloat16 *>(kp.dout.p) + elem_off(kp.dout, b, row_ok ? i : 0, h) + c0;
    const __nv_bfloat16 *k2 = reinterpret_cast<const __nv_bfloat16 *>(kp.k2.p) + c0;

#ifdef SA2_PROF
    long long seg_build = 0, seg_drain = 0;           // cycles after the waits of a build and of a fold
#endif
    // A_e = q_i * k2_{i-e} and B_e = dO_i * v2_{i-e} of sweep e.  Sixteen lanes take a row, 16 bytes each, so that a load
    // of the warp is whole rows: with a row per lane every load touched 32 cache lines, ~8000 cycles of L1 a sweep (10.3 -> 9.0 ms on
    // b1 n16384 h16; at head dim 64, without the rows in registers, 1.8 -> 2.2 ms on b4 n4096 h8).  The products are
    // formed before the wait for the stage, only the stores follow it.
    constexpr int LPR = D / 8, RPI = 32 / LPR;            // lanes per row, rows per load
    const int brow = (warp & 3) * 32 + lane / LPR, bcc = lane % LPR;
    const int64_t b_q = elem_off(kp.q, b, 0, h) + bcc * 8, b_do = elem_off(kp.dout, b, 0, h) + bcc * 8;
    const int64_t b_k2 = elem_off(kp.k2, b, 0, hk) + bcc * 8, b_v2 = elem_off(kp.v2, b, 0, hk) + bcc * 8;
    auto build = [&](int e) -> bool {
        auto fetch = [&](const TensorRef &t, int64_t base, int row) {
            return __ldg(reinterpret_cast<const uint4 *>(reinterpret_cast<const __nv_bfloat16 *>(t.p) + base + (int64_t)row * t.sn));
        };
        if constexpr (SPLIT) {
            // products and rests of four rows at a time, behind the wait: there are no registers to hold them before it
            if (e >= 1 && !warp_wait(&bars[BQ_AB_EMPTY], (e - 1) & 1, abort_flag, 3)) return false;
#pragma unroll 1
            for (int x0 = 0; x0 < LPR; x0 += 4) {
                uint4 w[4][4];                            // q, k2, dO, v2 of each row
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int ii = g.i0 + brow + (x0 + x) * RPI, kk = ii + kp.off2 - g.e0 - e;
                    const bool ok = ii < kp.n && kk >= 0;
                    w[x][0] = ok ? fetch(kp.q, b_q, ii) : make_uint4(0u, 0u, 0u, 0u);
                    w[x][1] = ok ? fetch(kp.k2, b_k2, kk) : make_uint4(0u, 0u, 0u, 0u);
                    w[x][2] = ok ? fetch(kp.dout, b_do, ii) : make_uint4(0u, 0u, 0u, 0u);
                    w[x][3] = ok ? fetch(kp.v2, b_v2, kk) : make_uint4(0u, 0u, 0u, 0u);
                }
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const uint32_t o = (bcc >> 3) * C::BLK + sw128_offset(brow + (x0 + x) * RPI, bcc & 7);
                    const uint4 a = mul_bf16x8(w[x][0], w[x][1]), b2 = mul_bf16x8(w[x][2], w[x][3]);
                    *reinterpret_cast<uint4 *>(sA + o) = a;
                    *reinterpret_cast<uint4 *>(sB + o) = b2;
                    *reinterpret_cast<uint4 *>(sA + C::REST + o) = mul_rest_bf16x8(w[x][0], w[x][1], a);
                    *reinterpret_cast<uint4 *>(sB + C::REST + o) = mul_rest_bf16x8(w[x][2], w[x][3], b2);
                }
            }
            fence_proxy_async_smem();
            mbar_arrive(&bars[BQ_AB_FULL]);
            return true;
        }
        uint4 pa[LPR], pb[LPR];
        constexpr int STEP = 2;                           // rows per lane that hold registers for a second operand
#pragma unroll
        for (int x0 = 0; x0 < LPR; x0 += STEP) {
            uint4 y[STEP];
#pragma unroll
            for (int x = 0; x < STEP; ++x) {
                const int ii = g.i0 + brow + (x0 + x) * RPI, kk = ii + kp.off2 - g.e0 - e;
                const bool ok = ii < kp.n && kk >= 0;
                pa[x0 + x] = ok ? fetch(kp.q, b_q, ii) : make_uint4(0u, 0u, 0u, 0u);
                y[x] = ok ? fetch(kp.k2, b_k2, kk) : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int x = 0; x < STEP; ++x) pa[x0 + x] = mul_bf16x8(pa[x0 + x], y[x]);
        }
#pragma unroll
        for (int x0 = 0; x0 < LPR; x0 += STEP) {
            uint4 y[STEP];
#pragma unroll
            for (int x = 0; x < STEP; ++x) {
                const int ii = g.i0 + brow + (x0 + x) * RPI, kk = ii + kp.off2 - g.e0 - e;
                const bool ok = ii < kp.n && kk >= 0;
                pb[x0 + x] = ok ? fetch(kp.dout, b_do, ii) : make_uint4(0u, 0u, 0u, 0u);
                y[x] = ok ? fetch(kp.v2, b_v2, kk) : make_uint4(0u, 0u, 0u, 0u);
            }
#pragma unroll
            for (int x = 0; x < STEP; ++x) pb[x0 + x] = mul_bf16x8(pb[x0 + x], y[x]);
        }
        if (e >= 1 && !warp_wait(&bars[BQ_AB_EMPTY], (e - 1) & 1, abort_flag, 3)) return false;
#ifdef SA2_PROF
        const long long seg_t0 = clock64();
#endif
#pragma unroll
        for (int x = 0; x < LPR; ++x) {
            const uint32_t o = (bcc >> 3) * C::BLK + sw128_offset(brow + x * RPI, bcc & 7);
            *reinterpret_cast<uint4 *>(sA + o) = pa[x];
            *reinterpret_cast<uint4 *>(sB + o) = pb[x];
        }
        fence_proxy_async_smem();
        mbar_arrive(&bars[BQ_AB_FULL]);
#ifdef SA2_PROF
        seg_build += clock64() - seg_t0;
#endif
        return true;
    };

    auto drain = [&](int v) -> bool {
        const int wb = v % C::UWBUF, e = v;
        const int kk = i + kp.off2 - g.e0 - e;
        const bool ok = row_ok && kk >= 0;
        // the first half of the k2 row is fetched before the wait, so that its latency overlaps the end of the
        // sweep; the second half with U
        const __nv_bfloat16 *kr = k2 + elem_off(kp.k2, b, ok ? kk : 0, hk);
        uint4 k2r[4];
#pragma unroll
        for (int cc = 0; cc < 4; ++cc) k2r[cc] = ok ? __ldg(reinterpret_cast<const uint4 *>(kr + cc * 8)) : make_uint4(0u, 0u, 0u, 0u);
        if (!warp_wait(&bars[BQ_W_FULL + wb], (v / C::UWBUF) & 1, abort_flag, 1)) return false;
        // A row of the shared accumulators is written by thread r in this sweep and by another thread in the
        // last one: every fold thread must have finished that one first.
        if (v >= 1 && !warp_wait(&bars[BQ_FOLD_SYNC], (v - 1) & 1, abort_flag, 2)) return false;
        tc_fence_after();
#ifdef SA2_PROF
        const long long seg_t0 = clock64();
#endif
        const int arow = r + P.epc - 1 - e;           // slab row of this thread in this sweep
        const bool fresh = e == 0 || r == 0;          // nothing has been added to the row yet
        if (v >= 1 && warp == 12) {
            // the top row of the last sweep is complete: it goes to the slab before thread 0 reuses its place
            const int trow = TQ - 1 + P.epc - e, arr = lane >> 4, c4 = (lane & 15) * 4;
            const float4 t = *reinterpret_cast<const float4 *>((arr ? acc_v : acc_k) + BqAcc<D>::off(trow, c4));
            *reinterpret_cast<float4 *>(slab + ((size_t)arr * (127 + P.epc) + trow) * D + c4) = t;
            __syncwarp();
        }
        // eight channels of one accumulator row += t * x (t: fp32 words, x: bf16; nothing where this thread has no row)
        auto rmw8 = [&](float *acc, int col, const uint32_t *t, const uint4 &x) {
            // both 16-byte pieces are read before either is written: the swizzled addresses hide from the
            // compiler that they are distinct, and it would order the second read after the first write
            ulonglong2 *p0 = reinterpret_cast<ulonglong2 *>(acc + BqAcc<D>::off(arow, col));
            ulonglong2 *p1 = reinterpret_cast<ulonglong2 *>(acc + BqAcc<D>::off(arow, col + 4));
            ulonglong2 t0 = {0, 0}, t1 = {0, 0};
            if (!fresh) { t0 = *p0; t1 = *p1; }
            if (ok) {
                t0.x = f2_fma(f2_pack(t[0], t[1]), f2_from_bf16x2(x.x), t0.x);
                t0.y = f2_fma(f2_pack(t[2], t[3]), f2_from_bf16x2(x.y), t0.y);
                t1.x = f2_fma(f2_pack(t[4], t[5]), f2_from_bf16x2(x.z), t1.x);
                t1.y = f2_fma(f2_pack(t[6], t[7]), f2_from_bf16x2(x.w), t1.y);
            }
            *p0 = t0;
            *p1 = t1;
        };
        // W first, then U, 32 channels at a time: only 32 registers of U / W are live at once, which keeps this
        // group within its budget without spills (the accumulator pair is released after the last read).
        {
            uint4 dr[NC];
#pragma unroll
            for (int c8 = 0; c8 < NC; ++c8) dr[c8] = __ldg(reinterpret_cast<const uint4 *>(dorow + c8 * 8));
#pragma unroll
            for (int hf = 0; hf < C::CC / 32; ++hf) {
                uint32_t w[32];
                tmem_ld32(lane_addr + C::UW0 + wb * 128 + 64 + hf * 32, w);
                tmem_wait_ld();
                // (a row is written even when this thread has nothing to add)
#pragma unroll
                for (int c4 = 0; c4 < 4; ++c4) rmw8(acc_v, (hf * 4 + c4) * 8, w + c4 * 8, dr[hf * 4 + c4]);
            }
        }
        {
            uint4 qr[NC];
#pragma unroll
            for (int c8 = 0; c8 < NC; ++c8) qr[c8] = __ldg(reinterpret_cast<const uint4 *>(qrow + c8 * 8));
#pragma unroll
            for (int hf = 0; hf < C::CC / 32; ++hf) {
                uint32_t u[32];
                tmem_ld32(lane_addr + C::UW0 + wb * 128 + hf * 32, u);
                if (hf == 1) {
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc)
                        k2r[cc] = ok ? __ldg(reinterpret_cast<const uint4 *>(kr + 32 + cc * 8)) : make_uint4(0u, 0u, 0u, 0u);
                }
                tmem_wait_ld();
                if (hf == C::CC / 32 - 1) {
                    // U and W of the sweep are in registers (or already used): the tensor cores may overwrite them
                    tc_fence_before();
                    mbar_arrive(&bars[BQ_W_EMPTY + wb]);
                }
#pragma unroll
                for (int c4 = 0; c4 < 4; ++c4) {
                    const int c8 = hf * 4 + c4;
                    const uint32_t kw[4] = {k2r[c4].x, k2r[c4].y, k2r[c4].z, k2r[c4].w};       // zero without a row
#pragma unroll
                    for (int z = 0; z < 4; ++z)
                        dq[c8 * 4 + z] = f2_fma(f2_pack(u[c4 * 8 + 2 * z], u[c4 * 8 + 2 * z + 1]), f2_from_bf16x2(kw[z]), dq[c8 * 4 + z]);
                    rmw8(acc_k, c8 * 8, u + c4 * 8, qr[c8]);
                }
            }
        }
        mbar_arrive(&bars[BQ_FOLD_SYNC]);
#ifdef SA2_PROF
        seg_drain += clock64() - seg_t0;
#endif
        return true;
    };

    const int nv = g.total > 0 ? g.nsweeps : 0;       // a split whose tiles all lie before the sequence start has no work
    int err = 0;
    if (nv > 0 && !build(0)) err = ERR_BQ_COMPUTE;
    for (int v = 0; v < nv && err == 0; ++v) {
        // the operands of the next sweep first: the tensor cores wait for them, U / W of this sweep arrive later
        if (v + 1 < nv && !build(v + 1)) { err = ERR_BQ_COMPUTE; break; }
        if (!drain(v)) err = ERR_BQ_COMPUTE;
    }

    SA2_PROF_ADD(4, seg_build);
    SA2_PROF_ADD(5, seg_drain);
    if (row_ok) bq_store_dq<D>(P, g, i, dq, err != 0 || *abort_flag != 0);
    return err;
}

// A fold group: WHICH = 0 U (head dim 128: both), 1 W.
template <int D, bool SPLIT, int WHICH>
__device__ __forceinline__ int bq_fold(const BqParams &P, const BqGeom &g, uint32_t tmem, float *acc_k, float *acc_v, uint8_t *sA, uint8_t *sB,
                                       uint64_t *bars, volatile int *abort_flag) {
    using C = BqCfg<D, SPLIT>;
    const KernelParams &kp = P.kp;
    const int ft = threadIdx.x & 127;
    const int h = blockIdx.y, b = blockIdx.z;
    const int slab_rows = 127 + P.epc;
    // this CTA's 64 channels of its slab (dK2 rows, then dV2 rows)
    float *slab = P.part_k2 + ((((size_t)b * kp.hq + h) * P.nqt + g.qt) * P.nsplit + g.split) * (size_t)(2 * slab_rows * D) + g.chh * 64;
    int err;
    if constexpr (C::TWO_FOLDS) {
        float *acc = WHICH ? acc_v : acc_k;
        for (int x = ft; x < slab_rows * BQ_ACC_STRIDE; x += 128) acc[x] = 0.f;      // only this group touches it
        bq_fold_sync(WHICH);
        err = bq_fold_half<D, SPLIT, WHICH>(P, g, tmem, acc, WHICH ? sB : sA, bars, abort_flag);
    } else {
        err = bq_fold_body<D, SPLIT>(P, g, tmem, acc_k, acc_v, slab, sA, sB, bars, abort_flag);
    }
    // The barrier sits outside the body so that a warp that gave up on a wait still reaches it.
    bq_fold_sync(WHICH);
    // Ring: rows above the live ones went to the slab when they were completed; the live rows follow now, and
    // the rows below them (second keys before the sequence start, when fewer than w2 sweeps ran) are zero.
    const int nv = g.total > 0 ? g.nsweeps : 0;
    const int live0 = BqAcc<D>::RING ? P.epc - nv : 0;                 // first slab row held in shared memory
    const int rows = BqAcc<D>::RING && nv > 0 ? live0 + BQ_ACC_RING : slab_rows;
    const bool held = !BqAcc<D>::RING || nv > 0;
    const bool bad = err != 0 || *abort_flag != 0;     // a CTA in which a wait ran out reports NaN
    constexpr int C4 = C::CC / 4;
    for (int x = ft; x < (C::TWO_FOLDS ? 1 : 2) * rows * C4; x += 128) {
        const int arr = C::TWO_FOLDS ? WHICH : x / (rows * C4), y = C::TWO_FOLDS ? x : x - arr * rows * C4;
        const int row = y / C4, c4 = (y % C4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (held && row >= live0) v = *reinterpret_cast<const float4 *>((arr ? acc_v : acc_k) + BqAcc<D>::off(row, c4));
        if (bad) v = make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F);
        *reinterpret_cast<float4 *>(slab + ((size_t)arr * slab_rows + row) * D + c4) = v;
    }
    return err;
}

template <int D, bool SPLIT>
__global__ void __launch_bounds__(BqCfg<D, SPLIT>::THREADS, 1)
bwd_q_kernel(const __grid_constant__ CUtensorMap mapK, const __grid_constant__ CUtensorMap mapV, const BqParams P) {
    using C = BqCfg<D, SPLIT>;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = align_smem(smem_raw);
    uint8_t *sK = smem;
    uint8_t *sV = sK + C::KV_BYTES;
    uint8_t *sA = sV + C::KV_BYTES;
    uint8_t *sB = sA + C::TILE;
    float *acc_k = reinterpret_cast<float *>(sB + C::TILE);
    const int acc_floats = BqAcc<D>::rows(P.epc) * BqAcc<D>::row_floats();
    float *acc_v = acc_k + acc_floats;
    uint64_t *bars = reinterpret_cast<uint64_t *>(acc_v + acc_floats);
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bars + BQ_BAR_COUNT);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_holder + 1);

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);       // warp-uniform, and known to be
    if (threadIdx.x == 0) {
        for (int x = 0; x < BQ_BAR_COUNT; ++x) {
            const bool pfull = x >= BQ_P_FULL && x < BQ_P_FULL + 3;          // every compute thread
            const bool fold = (x >= BQ_W_EMPTY && x < BQ_W_EMPTY + 2) || (x >= BQ_FOLD_SYNC && x < BQ_FOLD_SYNC + 2) ||
                              (x >= BQ_AB_FULL && x < BQ_AB_FULL + 2);      // every thread of a fold group
            // S_FULL collects a commit from each of the two first-product issuers, G_DONE (two folds) from each of
            // the two second-product issuers; AB_EMPTY from both issuers where A and B share it
            const bool two = (x >= BQ_S_FULL && x < BQ_S_FULL + 3) || (C::TWO_FOLDS ? x >= BQ_G_DONE && x < BQ_G_DONE + 3 : x == BQ_AB_EMPTY);
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
    const BqGeom g = bq_geom<D>(P);

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
        // of a scheduler then hold once
        reg_dealloc<C::REGS_COMPUTE>();
        err = bq_compute<D, SPLIT>(P, g, (warp >> 2) - 1, tmem, bars, abort_flag);
    } else if (!C::TWO_FOLDS || warp < 16) {
        reg_alloc<C::REGS_FOLD>();
        err = bq_fold<D, SPLIT, 0>(P, g, tmem, acc_k, acc_v, sA, sB, bars, abort_flag);
    } else if constexpr (C::TWO_FOLDS) {
        reg_alloc<C::REGS_FOLD_W>();
        err = bq_fold<D, SPLIT, 1>(P, g, tmem, acc_k, acc_v, sA, sB, bars, abort_flag);
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
// T and the split of offsets [e0, e0 + epc) at slab row k - off2 - 128 T + e0 + epc - 1, for the
// one or two tiles where that index falls inside [0, 127 + epc).
// ---------------------------------------------------------------------------
template <int D>
__global__ void bwd_q_reduce_kernel(const BqParams P) {
    constexpr int TPR = D / 4;                          // threads per row
    const KernelParams &kp = P.kp;
    const int acc_rows = 127 + P.epc;
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
        for (int hh = 0; hh < kp.g; ++hh) {
            const int h = hk * kp.g + hh;
            for (int s = 0; s < P.nsplit; ++s) {
                // tiles T with 0 <= pos - 128 T + top < acc_rows
                const int top = (s / P.tsplit) * P.epc + P.epc - 1;
                const int t_hi = min(P.nqt - 1, pos + top >= 0 ? (pos + top) / TQ : -1);
                for (int T = max(0, t_hi - 1); T <= t_hi; ++T) {
                    const int row = pos - TQ * T + top;
                    if (row < 0 || row >= acc_rows) continue;
                    const float *slab = P.part_k2 + ((((size_t)b * kp.hq + h) * P.nqt + T) * P.nsplit + s) * (size_t)(2 * acc_rows * D);
                    const float4 vk = *reinterpret_cast<const float4 *>(slab + (size_t)row * D + c4);
                    const float4 vv = *reinterpret_cast<const float4 *>(slab + (size_t)(acc_rows + row) * D + c4);
                    ak[0] += vk.x; ak[1] += vk.y; ak[2] += vk.z; ak[3] += vk.w;
                    av[0] += vv.x; av[1] += vv.y; av[2] += vv.z; av[3] += vv.w;
                }
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
