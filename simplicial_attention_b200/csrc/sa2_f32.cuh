// Host side of the fp32 kernels on the tensor cores: which calls they take, splits, scratch, launches.
#pragma once
#include "sa2.h"
#include "sa2_f32_fwd.cuh"
#include "sa2_f32_bwd.cuh"
#include "sa2_simt.cuh"
#include <algorithm>
#include <atomic>

namespace sa2 {
namespace f32 {

// fp32 tensors at head dims 32 and 64, any window, any strides the ABI takes.  (Head dim 128: the three terms of A_e, B_e and of
// a unit of K1 and V1 do not fit the shared memory of an SM.)
inline bool supported(const sa2_shape &s) { return s.kernel == SA2_KERNEL_AUTO && s.dtype == SA2_F32 && s.d <= 64; }

// Clusters of sixteen CTAs are the device's choice (at one CTA per SM they take most of a GPC): asked for once per device.
template <int D> inline bool sixteen_fit() {
    static std::atomic<int> known[64];             // 0: not asked yet, 1: no, 2: yes
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return false;
    int k = known[dev].load(std::memory_order_relaxed);
    if (k == 0) {
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 16; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
        cfg.gridDim = dim3(16); cfg.blockDim = dim3(FWD_THREADS); cfg.dynamicSmemBytes = fwd_smem_bytes<D>();
        cfg.attrs = &attr; cfg.numAttrs = 1;
        int n = 0;
        const bool ok = cudaFuncSetAttribute(fwd_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fwd_smem_bytes<D>()) == cudaSuccess &&
                        cudaFuncSetAttribute(fwd_kernel<D>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                        cudaOccupancyMaxActiveClusters(&n, fwd_kernel<D>, &cfg) == cudaSuccess && n >= 2;
        if (!ok) (void)cudaGetLastError();
        k = ok ? 2 : 1;
        known[dev].store(k, std::memory_order_relaxed);
    }
    return k == 2;
}
// CTAs of a row tile (see simt::cluster_size); sixteen where eight leave most of the chip idle and each still has two pairs of offsets.
template <int D> inline int fwd(const KernelParams &kp, int *status, int sms, cudaStream_t st) {
    const int tiles = (kp.n + ROWS - 1) / ROWS;
    int ce = simt::cluster_size((int64_t)tiles * kp.hq, kp.w2, 2, sms);
    if (ce == 8 && (int64_t)tiles * kp.hq * 32 <= sms && kp.w2 >= 64 && sixteen_fit<D>()) ce = 16;
    return simt::launch_clusters(fwd_kernel<D>, dim3(tiles * ce, kp.hq, kp.b), FWD_THREADS, fwd_smem_bytes<D>(), ce, st, kp, status) &&
                   simt::launch_fwd<D>(kp, sms, st, true) ? SA2_OK : SA2_ERR_CUDA;
}

// Scratch after the D vector, for `round` batch elements at a time: an element that alone needs more than MOST runs on the scalar
// kernels, which need none (long second windows: the dQ slabs grow with n * w2).
constexpr size_t ROUND_BYTES = (size_t)256 << 20, MOST_BYTES = (size_t)1 << 30;

// Splits of a tile's work over CTAs: the query heads of its group (MODE_K1: pairs of one and a query unit) and the offsets.
// A unit takes ~4500 cycles, a CTA ~10000 of set-up and its results, a sweep of MODE_K2 ~2500 for its operands and its fold.
// Scratch is written and read again at ~2000 bytes a cycle: `part`, the bytes of one partial result, for every split (none if there is
// one), and MODE_K2's dQ slabs of 127 + epc rows, `row` bytes over all tiles and query heads, for every range of offsets.
// Splits whose scratch does not fit `room` are not looked at, except none: ranges of one or two offsets cost the slab of a whole tile each,
// and with groups of query heads that is most of the traffic.  (By the cost alone b1 n14406 hq16 hk2 d64 w507/31 took 31 ranges and 1.75 GB.)
struct Split { int hs, es, epc; };
inline size_t split_bytes(const Split &s, size_t part, size_t row) {
    return (s.hs * s.es > 1 ? s.hs * s.es * part : 0) + s.es * (size_t)(ROWS - 1 + s.epc) * row;
}
inline Split split(int64_t ctas, int heads, int w2, double per_offset, size_t part, size_t row, size_t room, int batch, int sms) {
    Split best{1, 1, w2};
    double best_cost = 0.;
    for (int hs = 1; hs <= heads && hs <= 16; ++hs)
        for (int es = 1; es <= w2 && hs * es <= 64; ++es) {
            const Split s{hs, es, (w2 + es - 1) / es};
            if ((w2 + s.epc - 1) / s.epc != es) continue;
            const size_t bytes = split_bytes(s, part, row);
            if (bytes > room && hs * es > 1) continue;
            const double one = 10000. + (double)((heads + hs - 1) / hs) * s.epc * per_offset;
            const double cost = tc::split_cost(ctas * hs * es, one, batch, sms) + (hs * es > 1 ? 3000. : 0.) + (double)bytes * batch / 2000.;
            if (best_cost == 0. || cost < tc::SPLIT_GAIN * best_cost) { best = s; best_cost = cost; }
        }
    return best;
}
inline int k2_tiles(const sa2_shape &s) { return (s.n + s.off2 + ROWS - 1) / ROWS; }
inline size_t part_bytes(const sa2_shape &s, int64_t rows) { return (size_t)rows * s.hk * 2 * s.d * sizeof(float); }
inline size_t slab_row_bytes(const sa2_shape &s) { return (size_t)s.hq * k2_tiles(s) * s.d * sizeof(float); }
inline Split split_k2(const sa2_shape &s, int batch, int sms) {
    const int keys = s.w1 + ROWS - 1 < s.n + s.off1 ? s.w1 + ROWS - 1 : s.n + s.off1;
    return split((int64_t)k2_tiles(s) * s.hk, s.hq / s.hk, s.w2, 2500. + (keys + UNIT - 1) / UNIT * 4500., part_bytes(s, (int64_t)k2_tiles(s) * ROWS),
                 slab_row_bytes(s), ROUND_BYTES, batch, sms);
}
inline Split split_k1(const sa2_shape &s, size_t room, int batch, int sms) {
    const int64_t tiles = (int64_t)((s.n + s.off1 + ROWS - 1) / ROWS) * s.hk;
    const int rows = s.w1 + ROWS - 1 < s.n ? s.w1 + ROWS - 1 : s.n;
    return split(tiles, s.hq / s.hk * ((rows + UNIT - 1) / UNIT), s.w2, 4500., part_bytes(s, tiles / s.hk * ROWS), 0, room, batch, sms);
}

struct Plan {
    bool tc;
    Split k1, k2;
    int tiles, round;
    size_t redo, slab, part2, part1;
};
inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
inline Plan plan(const sa2_shape &s, int whole_batch, int sms) {
    Plan p;
    p.k2 = split_k2(s, whole_batch, sms);
    const size_t slab = split_bytes(p.k2, 0, slab_row_bytes(s)), part2 = split_bytes(p.k2, part_bytes(s, s.n + s.off2), 0);
    p.k1 = split_k1(s, slab + part2 < ROUND_BYTES ? ROUND_BYTES - slab - part2 : 0, whole_batch, sms);
    p.tiles = k2_tiles(s);
    const size_t part1 = split_bytes(p.k1, part_bytes(s, s.n + s.off1), 0), one = slab + part2 + part1;
    p.tc = one <= MOST_BYTES;
    p.round = one * s.b <= ROUND_BYTES ? s.b : one > ROUND_BYTES ? 1 : (int)(ROUND_BYTES / one);
    p.redo = align256((size_t)2 * s.b * sizeof(int));
    p.slab = align256(slab * p.round);
    p.part2 = align256(part2 * p.round);
    p.part1 = align256(part1 * p.round);
    return p;
}
inline size_t bwd_workspace_bytes(const sa2_shape &s, int whole_batch, int sms) {
    const Plan p = plan(s, whole_batch, sms);
    return p.tc ? p.redo + p.slab + p.part2 + p.part1 : 0;
}
inline int bwd_launches(const sa2_shape &s, int whole_batch, int sms) {
    const Plan p = plan(s, whole_batch, sms);
    return p.tc ? 2 + 3 * ((s.b + p.round - 1) / p.round) : 2;
}

template <int D, int MODE> inline int bwd_launch(const BwdParams &P, int rows, cudaStream_t st) {
    if (cudaFuncSetAttribute(bwd_kernel<D, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bwd_smem_bytes<D, MODE>()) != cudaSuccess)
        return SA2_ERR_CUDA;
    bwd_kernel<D, MODE><<<dim3((rows + ROWS - 1) / ROWS * P.nsplit, P.kp.hk, P.kp.b), BwdCfg<MODE>::THREADS, bwd_smem_bytes<D, MODE>(), st>>>(P);
    return cudaGetLastError() == cudaSuccess ? SA2_OK : SA2_ERR_CUDA;
}
template <int D> inline int bwd(const KernelParams &all, const Plan &p, char *extra, int *status, int sms, cudaStream_t st, int phases) {
    if (phases == 0) phases = SA2_BWD_ROWSUM | SA2_BWD_K1 | SA2_BWD_Q;
    int *redo = reinterpret_cast<int *>(extra);
    if ((phases & SA2_BWD_ROWSUM) && !simt::launch_delta<D>(all, st, redo)) return SA2_ERR_CUDA;
    extra += p.redo;
    const bool k1 = phases & SA2_BWD_K1, k2 = phases & SA2_BWD_Q;
    for (int b0 = 0; (k1 || k2) && b0 < all.b; b0 += p.round) {
        const KernelParams kp = tc::batch_part(all, b0, all.b - b0 < p.round ? all.b - b0 : p.round);
        float *slab = reinterpret_cast<float *>(extra), *part2 = reinterpret_cast<float *>(extra + p.slab);
        float *part1 = reinterpret_cast<float *>(extra + p.slab + p.part2);
        const int n1 = p.k1.hs * p.k1.es, n2 = p.k2.hs * p.k2.es;
        if (k1)
            if (int e = bwd_launch<D, MODE_K1>({kp, n1, p.k1.hs, p.k1.epc, 0, part1, nullptr, redo + b0, status}, kp.nk1, st)) return e;
        if (k2)
            if (int e = bwd_launch<D, MODE_K2>({kp, n2, p.k2.hs, p.k2.epc, p.tiles, part2, slab, redo + all.b + b0, status}, kp.nk2, st)) return e;
        const ReduceParams R{kp, slab, part2, part1, p.tiles, p.k2.es, p.k2.epc, k2 && n2 > 1 ? n2 : 0, k1 && n1 > 1 ? n1 : 0, k2};
        const int64_t rows = (k2 ? (int64_t)kp.n * kp.hq : 0) + (R.k2_splits ? (int64_t)kp.nk2 * kp.hk : 0) + (R.k1_splits ? (int64_t)kp.nk1 * kp.hk : 0);
        if (rows == 0) continue;
        const int most = std::max(std::max(R.dq ? p.k2.es : 0, R.k2_splits), R.k1_splits);
        const int64_t threads = rows * kp.b * (D / 4);
        if (most >= 8) reduce_kernel<D, 8><<<(unsigned)((threads * 8 + 255) / 256), 256, 0, st>>>(R);
        else reduce_kernel<D, 1><<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(R);
        if (cudaGetLastError() != cudaSuccess) return SA2_ERR_CUDA;
    }
    if ((k1 || k2) && !simt::launch_bwd<D>(all, k2, k2, k1, sms, st, redo)) return SA2_ERR_CUDA;
    return SA2_OK;
}

}  // namespace f32
}  // namespace sa2
