// Host side of the tcgen05 / TMEM / TMA kernels (bf16 operands, fp32
// accumulation): applicability checks, tensor maps, launches.
#pragma once
#include "sa2.h"
#include "sa2_common.cuh"
#include "sa2_simt.cuh"
#include "sa2_tc_fwd.cuh"
#include "sa2_tc_bwd_k1.cuh"
#include "sa2_tc_bwd_q.cuh"
#include "sa2_tc_fwd128.cuh"
#include "sa2_tc_bwd_k1_128.cuh"
#include "sa2_tmap.cuh"
#include <algorithm>
#include <cstdlib>

namespace sa2 {
namespace tc {

constexpr int SM_COUNT = 148;     // B200

// The tensor-core forward handles bf16 at every head dim and any window.
inline bool fwd_supported(const sa2_shape &s) { return s.dtype == SA2_BF16; }
// Head dim 32, and head dim 64 with a first window of more than 513 rows (the caller's window, however short the sequence),
// keep the products q * k2 and the probabilities to 16 bits and more, as a bf16 value and a bf16 rest each, so that only
// the inputs and the result are rounded to 8 bits: callers of these shapes had fp32 arithmetic.  The products are exact
// that way.  Relative error of the output against 64 bits 1.57e-3 to 1.67e-3, as with fp32 arithmetic (2.2e-3 to 3.2e-3 with
// rounded operands); of the logsumexp 2e-6, absolute (3e-3 to 1.6e-2).
inline bool fwd_split(const sa2_shape &s) { return s.d == 32 || (s.d == 64 && s.w1 > 513); }
// So does the tensor-core backward (see bq_plan, and bwd_split for dK1 / dV1 at head dim 32).
inline bool bwd_supported(const sa2_shape &s) { return s.dtype == SA2_BF16; }
// A scale of (nearly) zero goes to the fp32 kernels: dK1/dV1 folds lse / scale into its products.
inline bool bwd_scale_ok(const sa2_shape &s) { return fabsf(s.scale) >= 1e-20f; }
inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
// CTAs sharing one query tile in the dQ/dK2/dV2 kernel: splits of the window (head dim 128 walks it in one CTA) times
// splits of the offsets (an even number each with pairs).  Head dim 128: a CTA costs ~12000 cycles of set-up, loads, slab and its share of
// the reduction, a 64-key unit of a sweep ~1700.  Up to head dim 64, fitted to b4 n3000 h8 with first windows of 64 to 512 rows and to b64 of
// 64 to 512 rows: set-up of a CTA, a sweep and its units, and the least a sweep takes.  Over these 78 shapes the tile that the model
// picks takes at most 3.4 % longer than the better one; pairs take up to 27 % longer in short windows, 128 rows up to 70 % in long ones.
struct BqCost { double setup, sweep, unit, least; };
inline BqCost bq_cost(int d, bool split, bool pair) {
    if (d == 32) return pair ? BqCost{11000., 2750., 980., 5000.} : BqCost{13400., 2320., 1010., 0.};
    if (split) return pair ? BqCost{13500., 5000., 1130., 7000.} : BqCost{19500., 3900., 1250., 0.};
    return pair ? BqCost{13500., 3572., 745., 5300.} : BqCost{19500., 2900., 790., 0.};
}
struct BqSplit { bool pair; int nu, ups, tsplit, esplit, epc; double cost; };
inline BqSplit bq_split(const sa2_shape &s, const BwdCaller &call, bool split, bool pair, int sms) {
    BqSplit r;
    r.pair = pair;
    const int rows = bq_rows(pair), step = bq_step(pair), have = (s.n + s.off1 + 63) / 64;
    const int max_units = split && s.d == 64 ? (pair ? BqCfg<64, true, true>::MAX_UNITS : BqCfg<64, true, false>::MAX_UNITS)
                                             : (pair ? BqCfg<64, false, true>::MAX_UNITS : BqCfg<64, false, false>::MAX_UNITS);
    r.nu = (s.w1 + rows - 1 + 63) / 64;
    r.tsplit = s.d == 128 ? 1 : (r.nu + max_units - 1) / max_units;
    r.ups = (r.nu + r.tsplit - 1) / r.tsplit;
    const int per = (std::min(r.nu, have) + r.tsplit - 1) / r.tsplit;
    const int64_t ctas = (int64_t)((s.n + rows - 1) / rows) * s.hq * r.tsplit;
    const int sweeps = (s.w2 + step - 1) / step, most = BQ_MAX_EPC / step, least = (sweeps + most - 1) / most;
    // What a sweep costs: half of the columns in partly masked units come for nothing (warps without a valid column skip them).
    const double rows_all = s.n, ramp = std::min(std::max(s.w1 - s.off1, 0), s.n);
    const double seen = (ramp * (2. * s.off1 + ramp + 1.) / 2. + (rows_all - ramp) * s.w1) / rows_all;           // keys of a row, on average
    const double units = (seen / 64. + rows / 128. * (1. - ramp / (2. * rows_all))) / r.tsplit;
    const BqCost c = bq_cost(s.d, split, pair);
    const double sweep = s.d == 128 ? per * 1700. : std::max(c.least, c.sweep + units * c.unit), setup = s.d == 128 ? 12000. : c.setup;
    r.cost = 0.;
    r.esplit = least;
    for (int es = least; es <= sweeps && (es <= 16 || es == least); ++es) {
        const double cost = split_cost(ctas * es, setup + (sweeps + es - 1) / es * sweep, call.batch, sms);
        if (r.cost == 0. || cost < SPLIT_GAIN * r.cost) { r.esplit = es; r.cost = cost; }
    }
    r.epc = (sweeps + r.esplit - 1) / r.esplit * step;
    r.esplit = (s.w2 + r.epc - 1) / r.epc;
    return r;
}
// How dQ, dK2 and dV2 are computed.  Up to 56 offsets (the caller's window, however short the sequence) head dims 64 and 128
// round A_e, B_e, P and G to bf16.  Callers of head dim 32 and of longer second windows had fp32 arithmetic: those keep 16 bits
// and more of each (BqCfg), and their gradients in bf16 are as far from 64 bits as those of the fp32 kernels.
// A long window is many ranges of 56 offsets, whose partials grow with w1 * w2.  The batch then goes through the scratch
// in rounds of at most BQ_ROUND_BYTES (one element at least); where one element needs more than BQ_MOST_BYTES, the fp32 kernels
// do it without any (b1 n4096 h8 d64 w4096/4096 would take 36 GB).
// Errors of dq, dk2, dv2 against 64 bits, n150...400: 1.9e-3 to 3.2e-3 as on the fp32 kernels, 2.3e-3 to 5.4e-3 with rounded
// operands.  (A round was twice as large when the slabs of a tile of 128 rows were.)
constexpr size_t BQ_ROUND_BYTES = (size_t)128 << 20, BQ_MOST_BYTES = (size_t)1 << 30;
struct BqPlan {
    bool tc, split;      // on the tensor cores; with rests
    BqSplit sp;
    int round;           // batch elements that share the scratch at a time
};
inline BqPlan bq_plan(const sa2_shape &s, const BwdCaller &call, int sms) {
    BqPlan p;
    const bool longer = call.w2 > BQ_FINE_W2;
    p.split = s.d == 32 || longer;
    p.sp = bq_split(s, call, p.split, true, sms);
    if (s.d <= 64) {
        const BqSplit rows = bq_split(s, call, p.split, false, sms);
        if (rows.cost < p.sp.cost) p.sp = rows;
    }
    p.round = s.b;
    p.tc = true;
    if (longer) {
        sa2_shape one = s;
        one.b = 1;
        const int ns = p.sp.tsplit * p.sp.esplit;
        const size_t bytes = bq_part_dq_bytes(one, ns) + bq_part_k2_bytes(one, bq_rows(p.sp.pair), ns, p.sp.epc);
        p.tc = bytes <= BQ_MOST_BYTES;
        if (bytes * s.b > BQ_ROUND_BYTES) p.round = bytes > BQ_ROUND_BYTES ? 1 : (int)(BQ_ROUND_BYTES / bytes);
    }
    return p;
}
// Diagnostic switch: SA2_MMA_N64=1 issues every head-dim-128 product over the channels as two N = 64
// instructions instead of one N = 128 instruction.
inline int n64_products() {
    static const int v = [] { const char *e = std::getenv("SA2_MMA_N64"); return (e && e[0] == '1') ? 1 : 0; }();
    return v;
}
// scratch after the D vector: per-split partial dQ, the per-CTA dK2/dV2 slabs, partial dK1/dV1
struct BwdScratch { size_t dq, k2, k1; };
inline BwdScratch bwd_scratch(const sa2_shape &s, const BwdCaller &call, const BqPlan &q) {
    const K1Split k1 = k1_split(s, call, SM_COUNT);
    BwdScratch b{0, 0, align256(k1_part_bytes(s, k1.si * k1.se))};
    if (q.tc) {
        sa2_shape r = s;
        r.b = q.round;
        const int ns = q.sp.tsplit * q.sp.esplit;
        b.dq = align256(bq_part_dq_bytes(r, ns));
        b.k2 = align256(bq_part_k2_bytes(r, bq_rows(q.sp.pair), ns, q.sp.epc));
    }
    return b;
}
inline size_t bwd_extra_workspace_bytes(const sa2_shape &s, const BwdCaller &call) {
    if (!bwd_supported(s)) return 0;
    const BwdScratch b = bwd_scratch(s, call, bq_plan(s, call, SM_COUNT));
    return b.dq + b.k2 + b.k1;
}
// forward: 1 kernel; backward: D = rowsum(O*dO), dK1/dV1, then dQ/dK2/dV2 and the reduction of the partials, per round
inline int launches(const sa2_shape &s, bool backward, const BwdCaller &call) {
    if (!backward) return 1;
    const BqPlan q = bq_plan(s, call, SM_COUNT);
    const K1Split k1 = k1_split(s, call, SM_COUNT);
    const int rounds = (s.b + q.round - 1) / q.round, k1_reduce = k1.si * k1.se > 1;
    return !q.tc ? 3 + k1_reduce : rounds == 1 ? 4 : 2 + 2 * rounds + k1_reduce;
}

inline bool tma_addressable(const TensorRef &t) {
    return (reinterpret_cast<uintptr_t>(t.p) & 15u) == 0 && t.sb % 8 == 0 && t.sn % 8 == 0 && t.sh % 8 == 0;
}

// Device status word (one per device): kernels OR error bits into it when a
// bounded wait expires.
__device__ int g_status_word;

inline int *status_word() {
    static int *ptrs[64] = {nullptr};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    if (!ptrs[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_status_word) != cudaSuccess) return nullptr;
        ptrs[dev] = reinterpret_cast<int *>(p);
    }
    return ptrs[dev];
}

// keys and values, which TMA loads: a tensor map cannot repeat a dimension (stride 0, an expanded tensor)
inline bool kv_addressable(const TensorRef &t, const KernelParams &kp, int rows) {
    return tma_addressable(t) && (t.sb != 0 || kp.b == 1) && (t.sn != 0 || rows == 1) && (t.sh != 0 || kp.hk == 1);
}
// 16-byte vector access and TMA need 16-byte aligned bases and strides that are multiples of 8 elements
inline bool fwd_addressable(const KernelParams &kp) {
    return kv_addressable(kp.k1, kp, kp.nk1) && kv_addressable(kp.v1, kp, kp.nk1) && kv_addressable(kp.k2, kp, kp.nk2) &&
           kv_addressable(kp.v2, kp, kp.nk2) && tma_addressable(kp.q) && tma_addressable(kp.out);
}

inline int fwd128(const KernelParams &kp, const sa2_shape &s, cudaStream_t st) {
    f128::Params P;
    P.kp = kp;
    P.ri_log2 = fwd_ri_log2(s, SM_COUNT);
    P.nslots = f128::SLOTS;
    P.win_boxes = f128::win_boxes(s.w2, P.ri_log2);
    P.c = s.scale * 1.4426950408889634f;
    P.pv_split = n64_products();
    P.status = status_word();
    if (!P.status) return SA2_ERR_CUDA;
    CUtensorMap mapK, mapV, mapV2;     // 64-row, 64-channel boxes; 32-row boxes of the second values
    if (!tmap::make_rows_map(&mapK, kp.k1.p, kp.b, kp.nk1, kp.hk, 128, kp.k1.sb, kp.k1.sn, kp.k1.sh, f128::UNIT) ||
        !tmap::make_rows_map(&mapV, kp.v1.p, kp.b, kp.nk1, kp.hk, 128, kp.v1.sb, kp.v1.sn, kp.v1.sh, f128::UNIT) ||
        !tmap::make_rows_map(&mapV2, kp.v2.p, kp.b, kp.nk2, kp.hk, 128, kp.v2.sb, kp.v2.sn, kp.v2.sh, 32))
        return SA2_ERR_CUDA;
    const size_t smem = f128::smem_bytes();
    if (cudaFuncSetAttribute(f128::fwd128_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return SA2_ERR_CUDA;
    const int ri = 1 << P.ri_log2;
    f128::fwd128_kernel<<<dim3((kp.n + ri - 1) / ri, kp.hq, kp.b), f128::THREADS, smem, st>>>(mapK, mapV, mapV2, P);
    return cudaGetLastError() == cudaSuccess ? SA2_OK : SA2_ERR_CUDA;
}

template <int D, bool SPLIT>
inline int fwd_launch(const KernelParams &kp, const sa2_shape &s, cudaStream_t st) {
    FwdParams P;
    P.kp = kp;
    P.ri_log2 = fwd_ri_log2(s, SM_COUNT);
    P.win_boxes = fwd_win_boxes(s.w2, P.ri_log2);
    constexpr int A_TILES = 2 * FwdA<D, SPLIT>::TILES;
    P.nslots = fwd_slots(s.w1, P.ri_log2, P.win_boxes, A_TILES);
    P.c = s.scale * 1.4426950408889634f;
    P.status = status_word();
    if (!P.status) return SA2_ERR_CUDA;
    CUtensorMap mapK, mapV, mapK2, mapV2;       // 64-row boxes of K1 / V1, 32-row boxes of the second keys / values
    if (!tmap::make_rows_map(&mapK, kp.k1.p, kp.b, kp.nk1, kp.hk, D, kp.k1.sb, kp.k1.sn, kp.k1.sh, FWD_UNIT) ||
        !tmap::make_rows_map(&mapV, kp.v1.p, kp.b, kp.nk1, kp.hk, D, kp.v1.sb, kp.v1.sn, kp.v1.sh, FWD_UNIT) ||
        !tmap::make_rows_map(&mapK2, kp.k2.p, kp.b, kp.nk2, kp.hk, D, kp.k2.sb, kp.k2.sn, kp.k2.sh, 32) ||
        !tmap::make_rows_map(&mapV2, kp.v2.p, kp.b, kp.nk2, kp.hk, D, kp.v2.sb, kp.v2.sn, kp.v2.sh, 32))
        return SA2_ERR_CUDA;
    const size_t smem = fwd_smem_bytes(P.nslots, P.win_boxes, A_TILES);
    if (cudaFuncSetAttribute(fwd_kernel<D, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return SA2_ERR_CUDA;
    const int ri = 1 << P.ri_log2;
    fwd_kernel<D, SPLIT><<<dim3((kp.n + ri - 1) / ri, kp.hq, kp.b), FWD_THREADS, smem, st>>>(mapK, mapV, mapK2, mapV2, P);
    return cudaGetLastError() == cudaSuccess ? SA2_OK : SA2_ERR_CUDA;
}

inline int fwd(const KernelParams &kp, const sa2_shape &s, bool split, cudaStream_t st) {
    if (!fwd_addressable(kp)) return SA2_ERR_INVALID;
    switch (s.d) {
        case 32: return fwd_launch<32, true>(kp, s, st);
        case 64: return split ? fwd_launch<64, true>(kp, s, st) : fwd_launch<64, false>(kp, s, st);
        default: return fwd128(kp, s, st);
    }
}

inline bool bwd_addressable(const KernelParams &kp) {
    return fwd_addressable(kp) && tma_addressable(kp.dout);
}

// dQ, dK2, dV2: query-tile-owned tcgen05 kernel
template <int D, bool SPLIT, bool PAIR>
inline int bwd_q_launch(const BqParams &Q, cudaStream_t st) {
    using C = BqCfg<D, SPLIT, PAIR>;
    const KernelParams &kp = Q.kp;
    const size_t smem = C::SMEM;
    if (cudaFuncSetAttribute(bwd_q_kernel<D, SPLIT, PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return SA2_ERR_CUDA;
    CUtensorMap mapK, mapV;             // units of 64 rows
    constexpr int ROWS = 64;
    if (!tmap::make_rows_map(&mapK, kp.k1.p, kp.b, kp.nk1, kp.hk, D, kp.k1.sb, kp.k1.sn, kp.k1.sh, ROWS) ||
        !tmap::make_rows_map(&mapV, kp.v1.p, kp.b, kp.nk1, kp.hk, D, kp.v1.sb, kp.v1.sn, kp.v1.sh, ROWS))
        return SA2_ERR_CUDA;
    bwd_q_kernel<D, SPLIT, PAIR><<<dim3(Q.nqt * Q.nsplit, kp.hq, kp.b), C::THREADS, smem, st>>>(mapK, mapV, Q);
    return cudaGetLastError() == cudaSuccess ? SA2_OK : SA2_ERR_CUDA;
}

// deterministic reduction of the partials
template <int D>
inline int bwd_reduce_launch(const BqParams &Q, bool pair, cudaStream_t st) {
    const KernelParams &kp = Q.kp;
    const int64_t rows = (Q.reduce_q ? (Q.nsplit == 1 ? 0 : (int64_t)kp.b * kp.n * kp.hq) + (int64_t)kp.b * kp.nk2 * kp.hk : 0) +
                         (Q.reduce_k1 ? (int64_t)kp.b * kp.nk1 * kp.hk : 0);
    if (rows == 0) return SA2_OK;
    const unsigned blocks = (unsigned)((rows * (D / 4) + 255) / 256);
    const bool grouped = kp.g > 1 && Q.nsplit == 1;
    if (D == 128 || pair) (grouped ? bwd_q_reduce_kernel<D, true, true> : bwd_q_reduce_kernel<D, true, false>)<<<blocks, 256, 0, st>>>(Q);
    else (grouped ? bwd_q_reduce_kernel<D, D == 128, true> : bwd_q_reduce_kernel<D, D == 128, false>)<<<blocks, 256, 0, st>>>(Q);
    return cudaGetLastError() == cudaSuccess ? SA2_OK : SA2_ERR_CUDA;
}

template <int D>
inline int bwd_k1_launch(const KernelParams &kp, const sa2_shape &s, const CUtensorMap &mapK, const CUtensorMap &mapV, float c, int *status,
                         const K1Split &sp, float *part, cudaStream_t st) {
    CUtensorMap mapK2, mapV2;      // second keys / values, 32-row boxes of 64 channels
    if (!tmap::make_rows_map(&mapK2, kp.k2.p, kp.b, kp.nk2, kp.hk, D, kp.k2.sb, kp.k2.sn, kp.k2.sh, 32) ||
        !tmap::make_rows_map(&mapV2, kp.v2.p, kp.b, kp.nk2, kp.hk, D, kp.v2.sb, kp.v2.sn, kp.v2.sh, 32))
        return SA2_ERR_CUDA;
    const int ce = sp.si * sp.se;
    const dim3 grid((kp.nk1 + TJ - 1) / TJ * ce, kp.hk, kp.b);
    if constexpr (D == 128) {
        k128::Params P;
        P.kp = kp; P.c = c; P.ce = ce; P.si = sp.si; P.epc = sp.epc; P.part = part; P.n_split = n64_products(); P.status = status;
        if (cudaFuncSetAttribute(k128::bwd_k1_128_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k128::smem_bytes()) != cudaSuccess)
            return SA2_ERR_CUDA;
        k128::bwd_k1_128_kernel<<<grid, k128::THREADS, k128::smem_bytes(), st>>>(mapK, mapV, mapK2, mapV2, P);
    } else {
        BwdParams P;
        P.kp = kp; P.c = c; P.ce = ce; P.si = sp.si; P.epc = sp.epc; P.part = part; P.status = status;
        if (cudaFuncSetAttribute(bwd_k1_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bk1_smem_bytes()) != cudaSuccess)
            return SA2_ERR_CUDA;
        bwd_k1_kernel<D><<<grid, BK1_THREADS, bk1_smem_bytes(), st>>>(mapK, mapV, mapK2, mapV2, P);
    }
    return cudaGetLastError() == cudaSuccess ? SA2_OK : SA2_ERR_CUDA;
}

// batch elements [b0, b0 + nb) of a backward
inline KernelParams batch_part(KernelParams kp, int b0, int nb) {
    auto shift = [b0](TensorRef &t, int bytes) { t.p = reinterpret_cast<char *>(t.p) + b0 * t.sb * bytes; };
    for (TensorRef *t : {&kp.q, &kp.k1, &kp.k2, &kp.v1, &kp.v2, &kp.out, &kp.dout}) shift(*t, kp.in_bf16 ? 2 : 4);
    for (TensorRef *t : {&kp.dq, &kp.dk1, &kp.dk2, &kp.dv1, &kp.dv2}) shift(*t, kp.grad_bf16 ? 2 : 4);
    kp.lse += (int64_t)b0 * kp.hq * kp.n;
    kp.delta += (int64_t)b0 * kp.hq * kp.n;
    kp.b = nb;
    return kp;
}

template <int D>
inline int bwd_launch(const KernelParams &kp, const sa2_shape &s, const BwdCaller &call, void *extra, cudaStream_t st, int phases) {
    const float c = s.scale * 1.4426950408889634f;
    int *status = status_word();
    if (!status) return SA2_ERR_CUDA;
    if (phases == 0) phases = SA2_BWD_ROWSUM | SA2_BWD_K1 | SA2_BWD_Q;
    // D_i = sum_c O_ic dO_ic
    if ((phases & SA2_BWD_ROWSUM) && !simt::launch_delta<D>(kp, st)) return SA2_ERR_CUDA;
    BqPlan plan = bq_plan(s, call, SM_COUNT);
    // fp32 gradients show the last bits, which AUTO leaves to the fp32 kernels
    if (s.kernel == SA2_KERNEL_AUTO && !kp.grad_bf16 && call.w2 > BQ_FINE_W2) plan.tc = false;
    const BwdScratch room = bwd_scratch(s, call, plan);
    const K1Split k1 = k1_split(s, call, SM_COUNT);
    BqParams Q;
    Q.kp = kp;
    Q.c = c;
    Q.nu = plan.sp.nu;
    Q.tsplit = plan.sp.tsplit;
    Q.nsplit = plan.sp.tsplit * plan.sp.esplit;
    Q.epc = plan.sp.epc;
    Q.units_per_split = plan.sp.ups;
    Q.nqt = (kp.n + bq_rows(plan.sp.pair) - 1) / bq_rows(plan.sp.pair);
    Q.part_dq = reinterpret_cast<float *>(extra);
    Q.part_k2 = reinterpret_cast<float *>(reinterpret_cast<char *>(extra) + room.dq);
    float *part_k1 = reinterpret_cast<float *>(reinterpret_cast<char *>(extra) + room.dq + room.k2);
    Q.part_k1 = part_k1;
    Q.status = status;
    Q.ce = k1.si * k1.se;
    const bool q_tc = (phases & SA2_BWD_Q) && plan.tc, k1_parts = (phases & SA2_BWD_K1) && Q.ce > 1;
    if (phases & SA2_BWD_K1) {
        CUtensorMap mapK, mapV;     // 128-row, 64-channel boxes of K1 / V1 (a head-dim-128 tile is two boxes)
        if (!tmap::make_rows_map(&mapK, kp.k1.p, kp.b, kp.nk1, kp.hk, D, kp.k1.sb, kp.k1.sn, kp.k1.sh, TJ) ||
            !tmap::make_rows_map(&mapV, kp.v1.p, kp.b, kp.nk1, kp.hk, D, kp.v1.sb, kp.v1.sn, kp.v1.sh, TJ))
            return SA2_ERR_CUDA;
        if (int e = bwd_k1_launch<D>(kp, s, mapK, mapV, c, status, k1, part_k1, st)) return e;
    }
    if ((phases & SA2_BWD_Q) && !plan.tc && !simt::launch_bwd<D>(kp, true, true, false, SM_COUNT, st)) return SA2_ERR_CUDA;
    const bool one_round = plan.round >= kp.b;
    for (int b0 = 0; q_tc && b0 < kp.b; b0 += plan.round) {
        Q.kp = batch_part(kp, b0, kp.b - b0 < plan.round ? kp.b - b0 : plan.round);
        const bool pair = D == 128 || plan.sp.pair;       // (tiles of 128 rows are not built for head dim 128)
        if (int e = D == 32 || plan.split ? (pair ? bwd_q_launch<D, true, true>(Q, st) : bwd_q_launch<D, true, D == 128>(Q, st))
                                          : (pair ? bwd_q_launch<D, D == 32, true>(Q, st) : bwd_q_launch<D, D == 32, D == 128>(Q, st)))
            return e;
        Q.reduce_q = 1;
        Q.reduce_k1 = one_round && k1_parts;
        if (int e = bwd_reduce_launch<D>(Q, plan.sp.pair, st)) return e;
    }
    if (!k1_parts || (q_tc && one_round)) return SA2_OK;
    Q.kp = kp;
    Q.reduce_q = 0;
    Q.reduce_k1 = 1;
    return bwd_reduce_launch<D>(Q, plan.sp.pair, st);
}

inline int bwd(const KernelParams &kp, const sa2_shape &s, const BwdCaller &call, void *extra, cudaStream_t st, int phases = 0) {
    if (!bwd_addressable(kp)) return SA2_ERR_INVALID;
    switch (s.d) {
        case 32: return bwd_launch<32>(kp, s, call, extra, st, phases);
        case 64: return bwd_launch<64>(kp, s, call, extra, st, phases);
        default: return bwd_launch<128>(kp, s, call, extra, st, phases);
    }
}

}  // namespace tc
}  // namespace sa2
