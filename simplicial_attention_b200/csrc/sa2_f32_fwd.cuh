// Forward of fp32 tensors on tcgen05 tensor cores, head dims 32 and 64 (operands of three bf16 terms, sa2_f32_common.cuh).
//
// A CTA owns 128 query rows of one (batch, query head) and walks pairs of offsets e = i - k, one for each of two softmax
// groups, against units of 64 keys:
//     S = A_e K1^T     P = exp2(S - ref)     W = P V1     O += v2_{i-e} * W        (A_e = scale log2(e) q_i * k2_{i-e})
// A thread of a group owns a row: it forms P and its terms over the columns of S, adds the W of the last unit to the sum of
// its sweep, and at the end of the sweep folds that into the row's output.  References move as in the scalar kernels.
// The pairs of offsets are dealt out to the CTAs of a cluster, whose partial outputs meet through distributed shared memory:
// a short sequence has few row tiles.
//
// Warps (512 threads): 0 and 1 issuers of the groups' products; 4-7 and 8-11 softmax groups; 12-15 builders of A_e and of the
// terms of K1 / V1 units (two slots).  An issuer's products complete in order, so one barrier says both that S of unit u is
// there and that W of unit u - 1 is.  TMEM: group x at 160 x: terms of P over S in 96 columns, W in 64; the rows'
// partial outputs at 320 + 64 x, touched once a sweep.
//
// Bound: the chain S -> P -> P V1 of a group: ~3600 cycles of a softmax warp a unit, then ~2200 of products (24 of each kind), during
// which the other group has the exponentials.  b1 n1024 h8 d64 w512/32 2.0 ms on the scalar kernels -> 0.29 ms; 0.37 without the
// turns (F_TURN), with or without the output in registers.
#pragma once
#include "sa2_f32_common.cuh"
#include <cooperative_groups.h>

namespace sa2 {
namespace f32 {

constexpr int FWD_THREADS = 512;
constexpr int FWD_REGS_LAUNCH = 128, FWD_REGS_ISSUE = 40, FWD_REGS_SOFTMAX = 168, FWD_REGS_BUILD = 136;
static_assert(FWD_REGS_ISSUE + 2 * FWD_REGS_SOFTMAX + FWD_REGS_BUILD == 4 * FWD_REGS_LAUNCH, "register pool must balance");

enum FwdBar {
    F_A_FULL = 0,      // [2] per group
    F_A_EMPTY = 2,     // [2]
    F_KV_FULL = 4,     // [2] per slot
    F_KV_EMPTY = 6,    // [2]
    F_S_FULL = 8,      // [2] per group: S of unit u and W of unit u - 1
    F_P_FULL = 10,     // [2]
    F_TURN = 12,       // [2] the other group's products of the unit have been issued
    F_BAR_COUNT = 14
};

template <int D> inline size_t fwd_smem_bytes() {
    return 1024 + 2 * Planes<D>::bytes(ROWS) + 4 * Planes<D>::bytes(UNIT) + 256;
}

struct FwdGeom {
    int i0, i_last;
    int j_lo, nunits;       // units of every sweep: keys [j_lo + 64 w, +64)
    int pair0, dpair, npairs;     // pairs of offsets of this CTA: pair0, pair0 + dpair, ...
    int limit;              // offsets any row of the tile has
};

__device__ __forceinline__ FwdGeom fwd_geom(const KernelParams &kp) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    FwdGeom g;
    g.dpair = (int)cl.num_blocks();
    g.pair0 = (int)cl.block_rank();
    g.i0 = (int)(blockIdx.x / g.dpair) * ROWS;
    g.i_last = min(g.i0 + ROWS - 1, kp.n - 1);
    g.j_lo = max(0, g.i0 + kp.off1 - kp.w1 + 1);
    g.nunits = (g.i_last + kp.off1 - g.j_lo) / UNIT + 1;
    g.limit = min(kp.w2, g.i_last + kp.off2 + 1);
    const int pairs = (g.limit + 1) / 2;
    g.npairs = pairs > g.pair0 ? (pairs - g.pair0 - 1) / g.dpair + 1 : 0;
    return g;
}

// issuer of group x: P V1 of the last unit, then S of the next one
template <int D>
__device__ __forceinline__ int fwd_issue(const FwdGeom &g, int x, uint32_t tmem, const uint8_t *sA, const uint8_t *sK, const uint8_t *sV,
                                         uint64_t *bars, volatile int *abort_flag) {
    const uint32_t s = tmem + x * 160 + LOGITS, p = tmem + x * 160, w = tmem + x * 160 + 96;
    const uint64_t dA = smem_desc_sw128(smem_u32(sA) + x * Planes<D>::bytes(ROWS));
    const uint64_t dK = smem_desc_sw128(smem_u32(sK)), dV = smem_desc_sw128(smem_u32(sV));
    constexpr uint32_t SLOT = Planes<D>::bytes(UNIT) >> 4;
    const int total = g.npairs * g.nunits;
    int u = 0;
    for (int pp = 0; pp < g.npairs; ++pp) {
        for (int k = 0; k < g.nunits; ++k, ++u) {
            if (u > 0 && !mbar_wait_warp(&bars[F_P_FULL + x], (u - 1) & 1, abort_flag, 0, 1)) return ERR_FWD;
            if (k == 0 && !mbar_wait_warp(&bars[F_A_FULL + x], pp & 1, abort_flag, 0, 2)) return ERR_FWD;
            if (!mbar_wait_warp(&bars[F_KV_FULL + (u & 1)], (u >> 1) & 1, abort_flag, 0, 3)) return ERR_FWD;
            // The groups take turns: left to themselves they fall into step, both on the tensor cores and then both on their exponentials.
            if ((x == 1 || u > 0) && !mbar_wait_warp(&bars[F_TURN + x], (x == 1 ? u : u - 1) & 1, abort_flag, 0, 4)) return ERR_FWD;
            tc_fence_after();
            if (elect_one()) {
                if (u > 0) {
                    issue_pv<D>(w, p, dV + ((u - 1) & 1) * SLOT);
                    tc_commit(&bars[F_KV_EMPTY + ((u - 1) & 1)]);
                }
                issue_nt<D>(s, dA, dK + (u & 1) * SLOT);
                tc_commit(&bars[F_S_FULL + x]);
                if (k == g.nunits - 1) tc_commit(&bars[F_A_EMPTY + x]);
                mbar_arrive(&bars[F_TURN + 1 - x]);
            }
        }
    }
    if (total > 0) {
        if (!mbar_wait_warp(&bars[F_P_FULL + x], (total - 1) & 1, abort_flag)) return ERR_FWD;
        tc_fence_after();
        if (elect_one()) {
            issue_pv<D>(w, p, dV + ((total - 1) & 1) * SLOT);
            tc_commit(&bars[F_S_FULL + x]);
        }
    }
    return 0;
}

// builders: K1 / V1 units, and A_e of both groups at the start of a pair of sweeps
template <int D>
__device__ __forceinline__ int fwd_build(const KernelParams &kp, const FwdGeom &g, uint8_t *sA, uint8_t *sK, uint8_t *sV, uint64_t *bars,
                                         volatile int *abort_flag, uint32_t *most) {
    constexpr int CPR = D / 8, RPP = 128 / CPR;          // chunks of a row, rows the builders cover at a time
    const int t = threadIdx.x & 127, c = t % CPR, r0 = t / CPR;
    const int h = blockIdx.y, b = blockIdx.z, hk = h / kp.g;
    const float mul = logit_factor(kp.scale, true);
    float most_a = 0.f, most_k = 0.f, most_v = 0.f;
    int u = 0;
    for (int pp = 0; pp < g.npairs; ++pp) {
        for (int w = 0; w < g.nunits; ++w, ++u) {
            const int j0 = g.j_lo + UNIT * w, slot = u & 1;
            uint8_t *dk = sK + slot * Planes<D>::bytes(UNIT), *dv = sV + slot * Planes<D>::bytes(UNIT);
            {
                constexpr int N = UNIT / RPP;
                float k[N][8], v[N][8];
#pragma unroll
                for (int y = 0; y < N; ++y) {
                    const int j = j0 + r0 + y * RPP;
                    const bool ok = j < kp.nk1;
                    load8(k[y], row_ptr(kp.k1, b, ok ? j : 0, hk) + c * 8, ok);
                    load8(v[y], row_ptr(kp.v1, b, ok ? j : 0, hk) + c * 8, ok);
                }
                if (u >= 2 && !warp_wait(&bars[F_KV_EMPTY + slot], ((u >> 1) - 1) & 1, abort_flag, 1)) return ERR_FWD;
#pragma unroll
                for (int y = 0; y < N; ++y) {
                    put8<D>(dk, UNIT, r0 + y * RPP, c, k[y], most_k);
                    put8<D>(dv, UNIT, r0 + y * RPP, c, v[y], most_v);
                }
            }
            fence_proxy_async_smem();
            mbar_arrive(&bars[F_KV_FULL + slot]);
            if (w > 0) continue;
#pragma unroll 1
            for (int x = 0; x < 2; ++x) {
                const int e = 2 * (g.pair0 + pp * g.dpair) + x;
                uint8_t *da = sA + x * Planes<D>::bytes(ROWS);
#pragma unroll 1
                for (int y0 = 0; y0 < ROWS / RPP; y0 += 4) {
                    float q[4][8], k2[4][8];
#pragma unroll
                    for (int y = 0; y < 4; ++y) {
                        const int i = g.i0 + r0 + (y0 + y) * RPP, k = i + kp.off2 - e;
                        const bool ok = i < kp.n && k >= 0 && e < kp.w2;
                        load8(q[y], row_ptr(kp.q, b, ok ? i : 0, h) + c * 8, ok);
                        load8(k2[y], row_ptr(kp.k2, b, ok ? k : 0, hk) + c * 8, ok);
                    }
                    if (y0 == 0 && pp > 0 && !warp_wait(&bars[F_A_EMPTY + x], (pp - 1) & 1, abort_flag, 2)) return ERR_FWD;
#pragma unroll
                    for (int y = 0; y < 4; ++y) {
#pragma unroll
                        for (int z = 0; z < 8; ++z) q[y][z] = mul * q[y][z] * k2[y][z];
                        put8<D>(da, ROWS, r0 + (y0 + y) * RPP, c, q[y], most_a);
                    }
                }
                fence_proxy_async_smem();
                mbar_arrive(&bars[F_A_FULL + x]);
            }
        }
    }
    put_most(&most[0], most_a);
    put_most(&most[1], most_k);
    put_most(&most[2], most_v);
    return 0;
}

// Softmax group x.  Leaves the row's partial output in TMEM (columns o) against the reference `ref`, with the denominator l; returns
// whether there is one through `any`.
template <int D>
__device__ __forceinline__ int fwd_softmax(const KernelParams &kp, const FwdGeom &g, int x, uint32_t tmem, uint32_t o, bool &any, float &ref, float &l,
                                           uint64_t *bars, volatile int *abort_flag) {
    const int r = threadIdx.x & 127;
    const uint32_t region = tmem + ((uint32_t)(r & 96) << 16) + x * 160;
    const int h = blockIdx.y, b = blockIdx.z, hk = h / kp.g;
    const int i = g.i0 + r;
    const bool row_ok = i < kp.n;
    uint64_t ws[D / 2];
#pragma unroll
    for (int z = 0; z < D / 2; ++z) ws[z] = 0;
    any = false;
    ref = -CUDART_INF_F;
    l = 0.f;
    // W of the unit before: to the sum of its sweep, and at the end of the sweep to the row
    auto collect = [&](bool last, int e) {
        add_acc<D>(region + 96, ws);
        if (!last) return;
        const int k = i + kp.off2 - e;
        const bool ok = row_ok && e < kp.w2 && k >= 0;
        const float4 *v2 = reinterpret_cast<const float4 *>(row_ptr(kp.v2, b, ok ? k : 0, hk));
#pragma unroll
        for (int c = 0; c < D; c += 32) {
            uint32_t t[32];
            if (any) {
                tmem_ld32(o + c, t);
                tmem_wait_ld(t);
            } else {
#pragma unroll
                for (int z = 0; z < 32; ++z) t[z] = 0u;
            }
            if (ok) {
#pragma unroll
                for (int z = 0; z < 8; ++z) {
                    const float4 v = __ldg(v2 + c / 4 + z);
                    float a[4];
                    f2_unpack(f2_fma(ws[c / 2 + 2 * z], f2_pack(v.x, v.y), f2_pack(t[4 * z], t[4 * z + 1])), a[0], a[1]);
                    f2_unpack(f2_fma(ws[c / 2 + 2 * z + 1], f2_pack(v.z, v.w), f2_pack(t[4 * z + 2], t[4 * z + 3])), a[2], a[3]);
#pragma unroll
                    for (int y = 0; y < 4; ++y) t[4 * z + y] = __float_as_uint(a[y]);
                }
            }
            tmem_st32(o + c, t);
        }
        tmem_wait_st();
        any = true;
#pragma unroll
        for (int z = 0; z < D / 2; ++z) ws[z] = 0;
    };
    int u = 0;
    for (int pp = 0; pp < g.npairs; ++pp) {
        const int e = 2 * (g.pair0 + pp * g.dpair) + x, k = i + kp.off2 - e;
        const bool sweep_ok = row_ok && e < kp.w2 && k >= 0;
        for (int w = 0; w < g.nunits; ++w, ++u) {
            const int j0 = g.j_lo + UNIT * w, d1 = i + kp.off1 - j0;
            int lo = max(0, d1 - kp.w1 + 1);
            const int hi = sweep_ok ? min(UNIT - 1, d1) : -1;
            uint32_t len;
            column_range(lo, hi, len);
            if (!warp_wait(&bars[F_S_FULL + x], u & 1, abort_flag, 1)) return ERR_FWD;
            tc_fence_after();
            if (u > 0) collect(w == 0, e - 2 * g.dpair);
            // sixteen columns at a time, either half from the outside in (put_terms)
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                const int kk = y < 2 ? y : 5 - y, c0 = 16 * kk;
                uint32_t s[16];
                // P of the columns against the reference; their sum
                auto probs = [&](bool full) -> float {
                    float s0 = 0.f, s1 = 0.f;
                    const uint64_t nref = f2_pack(-ref, -ref);
#pragma unroll
                    for (int z = 0; z < 16; z += 2) {
                        float a0, a1;
                        f2_unpack(f2_add(f2_pack(s[z], s[z + 1]), nref), a0, a1);
                        float p0 = ex2(a0), p1 = ex2(a1);
                        if (!full) {
                            p0 = (uint32_t)(c0 + z - lo) <= len ? p0 : 0.f;
                            p1 = (uint32_t)(c0 + z + 1 - lo) <= len ? p1 : 0.f;
                        }
                        s0 += p0; s1 += p1;
                        s[z] = __float_as_uint(p0); s[z + 1] = __float_as_uint(p1);
                    }
                    return s0 + s1;
                };
                if (__all_sync(0xffffffffu, lo > c0 + 15 || (int)(lo + len) < c0)) {       // nothing valid for this warp
#pragma unroll
                    for (int z = 0; z < 16; ++z) s[z] = 0u;
                } else {
                    tmem_ld16(region + LOGITS + c0, s);
                    tmem_wait_ld(s);
                    const bool full = __all_sync(0xffffffffu, lo <= c0 && (int)(lo + len) >= c0 + 15);
                    float sum = full ? probs(true) : probs(false);
                    if (__any_sync(0xffffffffu, !(sum <= 65536.f))) {
                        // a reference moves (always at a row's first keys)
                        tmem_ld16(region + LOGITS + c0, s);
                        tmem_wait_ld(s);
                        float mx = -CUDART_INF_F;
#pragma unroll
                        for (int z = 0; z < 16; ++z)
                            if ((uint32_t)(c0 + z - lo) <= len) mx = fmaxf(mx, __uint_as_float(s[z]));
                        float f = 1.f;
                        if (!(sum <= 65536.f) && mx > ref) {
                            f = ex2(ref - mx);                             // 0 on the first hit
                            ref = mx;
                            l *= f;
                            const uint64_t f2 = f2_pack(f, f);
#pragma unroll
                            for (int z = 0; z < D / 2; ++z) ws[z] = f2_mul(ws[z], f2);
                        }
                        if (__any_sync(0xffffffffu, f != 1.f)) {
                            // what was formed against the old one: the output, and this unit's columns so far
                            tmem_wait_st();
                            if (any)
#pragma unroll 1
                                for (int c = 0; c < D; c += 32) {
                                    uint32_t t[32];
                                    tmem_ld32(o + c, t);
                                    tmem_wait_ld(t);
#pragma unroll
                                    for (int z = 0; z < 32; ++z) t[z] = __float_as_uint(__uint_as_float(t[z]) * f);
                                    tmem_st32(o + c, t);
                                }
#pragma unroll 1
                            for (int before = 0; before < y; ++before) {
                                const int kb = before < 2 ? before : 5 - before;
                                uint32_t t[16];
                                get_terms(region, kb, t);
#pragma unroll
                                for (int z = 0; z < 16; ++z) t[z] = __float_as_uint(__uint_as_float(t[z]) * f);
                                put_terms(region, kb, t);
                            }
                            tmem_wait_st();
                        }
                        sum = probs(false);
                    }
                    l += sum;
                }
                put_terms(region, kk, s);
            }
            tmem_wait_st();
            tc_fence_before();
            mbar_arrive(&bars[F_P_FULL + x]);
        }
    }
    if (u > 0) {
        if (!warp_wait(&bars[F_S_FULL + x], u & 1, abort_flag, 1)) return ERR_FWD;
        tc_fence_after();
        collect(true, 2 * (g.pair0 + (g.npairs - 1) * g.dpair) + x);
    }
    return 0;
}

template <int D>
__global__ void __launch_bounds__(FWD_THREADS, 1) fwd_kernel(const KernelParams kp, int *status) {
    namespace cg = cooperative_groups;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = align_smem(smem_raw);
    uint8_t *sA = smem;                                           // A_e of either group
    uint8_t *sK = sA + 2 * Planes<D>::bytes(ROWS);                // two slots
    uint8_t *sV = sK + 2 * Planes<D>::bytes(UNIT);
    uint64_t *bars = reinterpret_cast<uint64_t *>(sV + 2 * Planes<D>::bytes(UNIT));
    uint32_t *tmem_holder = reinterpret_cast<uint32_t *>(bars + F_BAR_COUNT);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_holder + 1);
    uint32_t *most = tmem_holder + 2;                             // [3] largest magnitudes of A_e, K1, V1
    int *redo = reinterpret_cast<int *>(tmem_holder + 5);         // the tile is left to the scalar kernel

    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);
    if (threadIdx.x == 0) {
        for (int x = 0; x < F_BAR_COUNT; ++x) {
            const bool one = x == F_A_EMPTY || x == F_A_EMPTY + 1 || x == F_S_FULL || x == F_S_FULL + 1 || x >= F_TURN;
            const bool two = x == F_KV_EMPTY || x == F_KV_EMPTY + 1;
            mbar_init(&bars[x], one ? 1u : two ? 2u : 128u);
        }
        *abort_flag = 0;
        *redo = 0;
        most[0] = most[1] = most[2] = 0u;
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(tmem_holder, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_holder;
    const FwdGeom g = fwd_geom(kp);

    // the partial outputs of the groups lie over the operands: rows of D + 4 floats, then reference and denominator
    constexpr int LD = D + 4;
    float *part = reinterpret_cast<float *>(smem), *stats = part + 2 * ROWS * LD;
    int err = 0;
#ifdef SA2_PROF
    const long long prof_t0 = clock64();
    sa2::sm100::prof_begin();
#endif
    if (warp < 4) {
        reg_dealloc<FWD_REGS_ISSUE>();
        if (warp < 2) err = fwd_issue<D>(g, warp, tmem, sA, sK, sV, bars, abort_flag);
        tc_fence_before();
        __syncthreads();
    } else if (warp < 12) {
        reg_alloc<FWD_REGS_SOFTMAX>();
        const int x = (warp >> 2) - 1, r = threadIdx.x & 127;
        const uint32_t o = tmem + ((uint32_t)(r & 96) << 16) + 320 + 64 * x;
        float ref, l;
        bool any;
        err = fwd_softmax<D>(kp, g, x, tmem, o, any, ref, l, bars, abort_flag);
        const bool bad = __any_sync(0xffffffffu, err != 0) || *abort_flag != 0;
        tc_fence_before();
        __syncthreads();                  // no product reads the operands any more
        float *row = part + (x * ROWS + r) * LD;
        float top = fabsf(l);
#pragma unroll
        for (int c = 0; c < D; c += 32) {
            uint32_t t[32];
            tmem_ld32(o + c, t);
            tmem_wait_ld(t);
#pragma unroll
            for (int z = 0; z < 32; z += 2) asm("max.NaN.abs.f32 %0, %0, %1, %2;" : "+f"(top) : "f"(__uint_as_float(t[z])), "f"(__uint_as_float(t[z + 1])));
#pragma unroll
            for (int z = 0; z < 32; z += 4)
                *reinterpret_cast<float4 *>(row + c + z) =
                    bad ? make_float4(CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F, CUDART_NAN_F)
                        : !any ? make_float4(0.f, 0.f, 0.f, 0.f)
                               : make_float4(__uint_as_float(t[z]), __uint_as_float(t[z + 1]), __uint_as_float(t[z + 2]), __uint_as_float(t[z + 3]));
        }
        if (any && !bad && !(top <= CUDART_MAX_NORMAL_F)) *redo = 1;
        stats[(x * 2) * ROWS + r] = bad ? 0.f : ref;
        stats[(x * 2 + 1) * ROWS + r] = bad ? CUDART_NAN_F : l;
    } else {
        reg_alloc<FWD_REGS_BUILD>();
        err = fwd_build<D>(kp, g, sA, sK, sV, bars, abort_flag, most);
        tc_fence_before();
        __syncthreads();
        if ((threadIdx.x & 127) < 3 && out_of_range(__uint_as_float(most[threadIdx.x & 127]))) *redo = 1;
    }
    if (err) atomicOr(status, err);
    SA2_PROF_ADD(0, clock64() - prof_t0);
    SA2_PROF_END();
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    const int ce = (int)cl.num_blocks(), rows = ROWS / ce;
    for (int idx = threadIdx.x; idx < rows * (D / 4); idx += FWD_THREADS) {
        const int r = (int)cl.block_rank() * rows + idx / (D / 4), c = (idx % (D / 4)) * 4, i = g.i0 + r;
        if (i >= kp.n) continue;
        float *lse = kp.lse + ((int64_t)blockIdx.z * kp.hq + blockIdx.y) * kp.n + i;
        bool again = false;
        for (int q = 0; q < ce; ++q) again |= *cl.map_shared_rank(redo, q) != 0;
        if (again) {
            if (c == 0) *lse = __uint_as_float(LSE_REDO);
            continue;
        }
        float M = -CUDART_INF_F, L = 0.f, v[4] = {0.f, 0.f, 0.f, 0.f};
        for (int q = 0; q < 2 * ce; ++q) M = fmaxf(M, cl.map_shared_rank(stats, q >> 1)[(q & 1) * 2 * ROWS + r]);
        for (int q = 0; q < 2 * ce; ++q) {
            const float *st = cl.map_shared_rank(stats, q >> 1) + (q & 1) * 2 * ROWS;
            // (a group without a reference says nothing, or NaN where a wait ran out)
            if (!(st[r] > -CUDART_INF_F) && st[ROWS + r] == 0.f) continue;
            const float f = st[r] > -CUDART_INF_F ? ex2(st[r] - M) : 1.f;
            const float4 p = *reinterpret_cast<const float4 *>(cl.map_shared_rank(part, q >> 1) + ((q & 1) * ROWS + r) * LD + c);
            L = fmaf(st[ROWS + r], f, L);
            v[0] = fmaf(p.x, f, v[0]); v[1] = fmaf(p.y, f, v[1]); v[2] = fmaf(p.z, f, v[2]); v[3] = fmaf(p.w, f, v[3]);
        }
        const float inv = 1.f / L;
#pragma unroll
        for (int z = 0; z < 4; ++z) v[z] *= inv;
        store_vec<4>(kp.out.p, elem_off(kp.out, blockIdx.z, i, blockIdx.y) + c, false, v);
        if (c == 0) *lse = M * LN2 + __logf(L);
    }
    cl.sync();               // no CTA leaves while its shared memory is read
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

}  // namespace f32
}  // namespace sa2
