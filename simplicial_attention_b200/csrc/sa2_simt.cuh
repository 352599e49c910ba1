// fp32 SIMT kernels for sliding-window causal 2-simplicial attention.
//
// These are the exact-arithmetic tier: inputs (fp32 or bf16) are widened to
// fp32, every product and sum is fp32, and nothing is rounded to bf16 on the
// way.  They handle every head dim in {32, 64, 128}, any sequence length, any
// window and grouped-query heads, and they are the kernels the tensor-core
// path is checked against on the device.  fp32 tensors of head dims 32 and 64 come here only by request, without
// scratch, or where their backward needs more of it than is allowed; sa2_f32.cuh has them otherwise.
//
// Formulation ("k'-offset"): for an offset e = i - k in [0, w2) every query
// row i is paired with ONE second key k2[i-e].  A_e[i,:] = scale*q_i*k2_{i-e}
// turns the trilinear logits into an ordinary GEMM S_e = A_e K1^T, and
// W_e = P_e V1 followed by O += v2_{i-e} * W_e gives the output.  The softmax
// runs jointly over all (j, e).  The same tiles serve the three gradients:
//   rows = query rows i          -> dQ            (MODE_BWD_Q)
//   rows = second-key rows k=i-e -> dK2, dV2      (MODE_BWD_K2)
//   rows = first-key rows j      -> dK1, dV1      (MODE_BWD_K1, S^T tiles)
// Each output row is owned by one cluster of CTAs, so there are no atomics and
// results are bitwise reproducible.
//
// Tile: 64 rows x 64 columns by a group of 256 threads as a 16x16 grid; thread (ty, tx) owns rows ty+16*ii and
// columns tx+16*jj of the logit tile and rows ty+16*ii, channels tx*VEC.. of the accumulators.  The probabilities
// of a row are written and read by the same half-warp, so they need no barrier.
//
// A CTA holds two groups (one at head dim 128) that take alternate offsets against the same K1/V1 tiles, which
// stream through two buffers with cp.async; an offset's A (and B = dO * v2) tile is built once and used for the
// whole window.  The offsets of a row tile are further split over the CTAs of a cluster, whose accumulators are
// added (or merged, in the forward) through distributed shared memory: a short sequence has few row tiles, and
// walking all offsets one after the other left all but a few SMs idle.  The three gradients share one launch.
// Measured on a B200, against one CTA of 256 threads per row tile, three barriers a step and a launch per gradient:
// b1 n128 h2 d32 w128/128 forward + backward 5.0 -> 0.30 ms, b1 n1024 h8 d64 w512/32 11.8 -> 7.5 ms.
// Bound: issue slots - fp32 FMA are ~60 % of the instructions, and a scheduler issues one every other cycle.
#pragma once
#include "sa2_common.cuh"
#include <cooperative_groups.h>
#include <math_constants.h>

namespace sa2 {
namespace simt {

enum { MODE_FWD = 0, MODE_BWD_Q = 1, MODE_BWD_K2 = 2, MODE_BWD_K1 = 3 };

constexpr int TILE = 64;
constexpr int LP = TILE + 4;   // row stride of the probability tiles
constexpr int GROUP = 256;     // threads of a group
constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;

template <int D> struct Cfg {
    static constexpr int LD = D + 4;                 // row stride of [64][D] tiles
    static constexpr int CPT = D / 16;               // channels per thread
    static constexpr int VEC = (D >= 64) ? 4 : 2;    // vector width of a channel group
    static constexpr int NV = CPT / VEC;             // channel groups per thread
    static constexpr int NG = D == 128 ? 1 : 2;      // groups per CTA
    static constexpr int NBUF = D == 128 ? 1 : 2;    // K1/V1 tile buffers
    static constexpr int THREADS = NG * GROUP;
    static constexpr int TF = TILE * LD;             // floats of a [64][D] tile
    // K1/V1 buffers (reused by the final reduction: NG groups x 2 accumulators), then per group A, P (forward) or
    // A, B, P, G
    static constexpr size_t smem(bool bwd) {
        return sizeof(float) * (2 * NBUF * TF + NG * ((bwd ? 2 : 1) * TF + (bwd ? 2 : 1) * TILE * LP) + NG * 2 * TILE);
    }
};

// first channel of channel group u for thread column tx
template <int D> __device__ __forceinline__ int chan(int tx, int u) {
    return u * (16 * Cfg<D>::VEC) + tx * Cfg<D>::VEC;
}

__device__ __forceinline__ float ex2f(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// acc[ii][jj] = sum_c A[ty+16ii][c] * B[tx+16jj][c]
template <int D>
__device__ __forceinline__ void gemm_nt(const float *__restrict__ A, const float *__restrict__ B,
                                        int ty, int tx, float (&acc)[4][4]) {
    constexpr int LD = Cfg<D>::LD;
#pragma unroll
    for (int ii = 0; ii < 4; ++ii)
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) acc[ii][jj] = 0.f;
#pragma unroll 2
    for (int c = 0; c < D; c += 4) {
        float4 b[4];
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) b[jj] = *reinterpret_cast<const float4 *>(B + (tx + 16 * jj) * LD + c);
#pragma unroll
        for (int ii = 0; ii < 4; ++ii) {
            const float4 a = *reinterpret_cast<const float4 *>(A + (ty + 16 * ii) * LD + c);
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                acc[ii][jj] = fmaf(a.x, b[jj].x, acc[ii][jj]);
                acc[ii][jj] = fmaf(a.y, b[jj].y, acc[ii][jj]);
                acc[ii][jj] = fmaf(a.z, b[jj].z, acc[ii][jj]);
                acc[ii][jj] = fmaf(a.w, b[jj].w, acc[ii][jj]);
            }
        }
    }
}

// acc[ii][u*VEC+e] += sum_j P[ty+16ii][j] * X[j][chan(tx,u)+e]
template <int D>
__device__ __forceinline__ void gemm_pv(const float *__restrict__ P, const float *__restrict__ X,
                                        int ty, int tx, float (&acc)[4][Cfg<D>::CPT]) {
    constexpr int LD = Cfg<D>::LD, VEC = Cfg<D>::VEC, NV = Cfg<D>::NV;
#pragma unroll 1
    for (int j = 0; j < TILE; j += 4) {
        float4 pr[4];
#pragma unroll
        for (int ii = 0; ii < 4; ++ii) pr[ii] = *reinterpret_cast<const float4 *>(P + (ty + 16 * ii) * LP + j);
#pragma unroll
        for (int jj = 0; jj < 4; ++jj) {
#pragma unroll
            for (int u = 0; u < NV; ++u) {
                float x[VEC];
                load_vec<VEC>(X, (j + jj) * LD + chan<D>(tx, u), false, x);
#pragma unroll
                for (int ii = 0; ii < 4; ++ii) {
                    const float pv = jj == 0 ? pr[ii].x : jj == 1 ? pr[ii].y : jj == 2 ? pr[ii].z : pr[ii].w;
#pragma unroll
                    for (int e = 0; e < VEC; ++e) acc[ii][u * VEC + e] = fmaf(pv, x[e], acc[ii][u * VEC + e]);
                }
            }
        }
    }
}

// Start filling a [64][D] tile from rows row0.. of a tensor (zero outside [0, nrows)): asynchronous copies for fp32
// tensors (complete them with cp_wait), plain loads for bf16 ones.
template <int D>
__device__ __forceinline__ void fill_tile(float *S, const TensorRef &t, int b, int h, int row0, int nrows, bool bf16) {
    constexpr int LD = Cfg<D>::LD, C4 = D / 4;
    for (int idx = threadIdx.x; idx < TILE * C4; idx += Cfg<D>::THREADS) {
        const int r = idx / C4, c = (idx % C4) * 4, row = row0 + r;
        const bool ok = row >= 0 && row < nrows;
        if (!bf16) {
            const float *src = reinterpret_cast<const float *>(t.p) + elem_off(t, b, ok ? row : 0, h) + c;
            const uint32_t dst = (uint32_t)__cvta_generic_to_shared(S + r * LD + c);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
        } else {
            float v[4] = {0.f, 0.f, 0.f, 0.f};
            if (ok) load_vec<4>(t.p, elem_off(t, b, row, h) + c, true, v);
            *reinterpret_cast<float4 *>(S + r * LD + c) = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A[r][c] = mul * x[i(r)][c] * y[k(r)][c] for the 64 rows of a tile, by one group; rows whose (i, k) pair is invalid
// become zero.  i(r) = i_base + r, k(r) = k_base + r.
template <int D>
__device__ __forceinline__ void build_prod_tile(float *S, const TensorRef &x, int hx, const TensorRef &y, int hy,
                                                int b, int i_base, int n_i, int k_base, int n_k, float mul, bool bf16) {
    constexpr int LD = Cfg<D>::LD, C4 = D / 4;
#pragma unroll 4
    for (int idx = threadIdx.x & (GROUP - 1); idx < TILE * C4; idx += GROUP) {
        const int r = idx / C4, c = (idx % C4) * 4;
        const int i = i_base + r, k = k_base + r;
        float o[4] = {0.f, 0.f, 0.f, 0.f};
        if (i >= 0 && i < n_i && k >= 0 && k < n_k) {
            float a[4], e[4];
            load_vec<4>(x.p, elem_off(x, b, i, hx) + c, bf16, a);
            load_vec<4>(y.p, elem_off(y, b, k, hy) + c, bf16, e);
#pragma unroll
            for (int u = 0; u < 4; ++u) o[u] = mul * a[u] * e[u];
        }
        *reinterpret_cast<float4 *>(S + r * LD + c) = make_float4(o[0], o[1], o[2], o[3]);
    }
}

__device__ __forceinline__ float half_warp_max(float v) {
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float half_warp_sum(float v) {
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
// barrier of the 256 threads of a group
__device__ __forceinline__ void group_sync(int g) { asm volatile("bar.sync %0, 256;" ::"r"(g + 1) : "memory"); }

// Sums an accumulator over the groups of the CTAs of the cluster and stores the rows of this CTA's share:
// part[g] is group g's [64][D] tile at the same place in every CTA.
template <int D>
__device__ __forceinline__ void reduce_store(float *part, int tiles_apart, const TensorRef &dst, int b, int h, int row0, int nrows,
                                             float mul, bool bf16) {
    namespace cg = cooperative_groups;
    using C = Cfg<D>;
    cg::cluster_group cl = cg::this_cluster();
    const int ce = (int)cl.num_blocks(), rank = (int)cl.block_rank(), rows = TILE / ce;
    for (int idx = threadIdx.x; idx < rows * (D / 4); idx += C::THREADS) {
        const int r = rank * rows + idx / (D / 4), c = (idx % (D / 4)) * 4;
        if (row0 + r >= nrows) continue;
        float x[4] = {0.f, 0.f, 0.f, 0.f};
        for (int q = 0; q < ce; ++q) {
            const float *p = cl.map_shared_rank(part, q);
#pragma unroll
            for (int g = 0; g < C::NG; ++g) {
                const float4 v = *reinterpret_cast<const float4 *>(p + (size_t)g * tiles_apart * C::TF + r * C::LD + c);
                x[0] += v.x; x[1] += v.y; x[2] += v.z; x[3] += v.w;
            }
        }
#pragma unroll
        for (int z = 0; z < 4; ++z) x[z] *= mul;
        store_vec<4>(dst.p, elem_off(dst, b, row0 + r, h) + c, bf16, x);
    }
}
template <int D>
__device__ __forceinline__ void put_acc(float *tile, const float (&acc)[4][Cfg<D>::CPT], int ty, int tx) {
#pragma unroll
    for (int ii = 0; ii < 4; ++ii)
#pragma unroll
        for (int u = 0; u < Cfg<D>::NV; ++u) {
            float x[Cfg<D>::VEC];
#pragma unroll
            for (int q = 0; q < Cfg<D>::VEC; ++q) x[q] = acc[ii][u * Cfg<D>::VEC + q];
            store_vec<Cfg<D>::VEC>(tile, (ty + 16 * ii) * Cfg<D>::LD + chan<D>(tx, u), false, x);
        }
}

// The offsets are dealt out to the groups of the cluster's CTAs one by one: round x of group g in the CTA of rank r is
// offset (x * ce + r) * NG + g (the first offsets of a sequence see more rows than the last ones).
__device__ __forceinline__ void cluster_rank(int &ce, int &rank) {
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    ce = (int)cl.num_blocks();
    rank = (int)cl.block_rank();
}

// ---------------------------------------------------------------------------
// Row-owned tiles: forward, dQ, or dK2/dV2.  `tile`: row tile, `h_in`: query head (forward, dQ) or key/value head.
// ---------------------------------------------------------------------------
template <int D, int MODE>
__device__ __forceinline__ void row_tile(const KernelParams &p, float *smem, int tile, int h_in, int bi, bool redo) {
    namespace cg = cooperative_groups;
    using C = Cfg<D>;
    constexpr int CPT = C::CPT, VEC = C::VEC, NV = C::NV, TF = C::TF;
    constexpr bool BWD = MODE != MODE_FWD;
    const int grp = threadIdx.x / GROUP, t = threadIdx.x & (GROUP - 1), tx = t & 15, ty = t >> 4;
    float *KV = smem;                                            // [NBUF][K, V]
    float *own = KV + 2 * C::NBUF * TF + grp * ((BWD ? 2 : 1) * TF + (BWD ? 2 : 1) * TILE * LP);
    float *As = own, *Bs = As + TF, *Ps = own + (BWD ? 2 : 1) * TF, *Gs = Ps + TILE * LP;
    float *stats = KV + 2 * C::NBUF * TF + C::NG * ((BWD ? 2 : 1) * TF + (BWD ? 2 : 1) * TILE * LP);   // [NG][2][64]

    const int r0 = tile * TILE;
    const bool bf16 = p.in_bf16 != 0;
    const int hk_i = (MODE == MODE_BWD_K2) ? h_in : h_in / p.g;
    const int h_begin = (MODE == MODE_BWD_K2) ? hk_i * p.g : h_in;
    const int h_end = (MODE == MODE_BWD_K2) ? h_begin + p.g : h_begin + 1;
    int ce, rank;
    cluster_rank(ce, rank);

    float acc0[4][CPT];   // FWD: O   BWD_Q: dQ   BWD_K2: dK2
    float acc1[4][CPT];   // BWD_K2: dV2
    float ref[4], l_run[4];
#pragma unroll
    for (int ii = 0; ii < 4; ++ii) {
        ref[ii] = -CUDART_INF_F;
        l_run[ii] = 0.f;
#pragma unroll
        for (int c = 0; c < CPT; ++c) { acc0[ii][c] = 0.f; acc1[ii][c] = 0.f; }
    }

    for (int h = h_begin; h < h_end; ++h) {
        for (int ep = rank * C::NG; ep < p.w2; ep += ce * C::NG) {
            const int e = ep + grp;
            // rows of the tile for offset x: i = i_of(x) + r, k = k_of(x) + r; the valid ones are [ilo, ihi] in i
            auto i_of = [&](int x) { return MODE == MODE_BWD_K2 ? r0 - p.off2 + x : r0; };
            auto k_of = [&](int x) { return MODE == MODE_BWD_K2 ? r0 : r0 + p.off2 - x; };
            auto range = [&](int x, int &ilo, int &ihi) {
                const int ib = i_of(x), kb = k_of(x);
                ilo = max(ib, max(0, ib - kb));                          // i >= 0 and k >= 0
                ihi = min(min(ib + TILE - 1, p.n - 1), ib + (p.nk2 - 1 - kb));
            };
            // keys any of the CTA's groups needs in this round
            int j_lo = 1 << 30, j_hi = -1;
            for (int x = ep; x < min(ep + C::NG, p.w2); ++x) {
                int lo, hi;
                range(x, lo, hi);
                if (lo > hi) continue;
                j_lo = min(j_lo, max(0, lo + p.off1 - p.w1 + 1));
                j_hi = max(j_hi, hi + p.off1);
            }
            if (j_hi < 0) continue;
            const int i_base = i_of(e), k_base = k_of(e);
            int ilo = 1, ihi = 0;
            if (e < p.w2) range(e, ilo, ihi);
            const bool any = ilo <= ihi;

            __syncthreads();            // the last round's tiles are no longer read
            fill_tile<D>(KV, p.k1, bi, hk_i, j_lo, p.nk1, bf16);
            fill_tile<D>(KV + TF, p.v1, bi, hk_i, j_lo, p.nk1, bf16);
            cp_commit();
            if (any) {
                build_prod_tile<D>(As, p.q, h, p.k2, hk_i, bi, i_base, p.n, k_base, p.nk2, logit_factor(p.scale, redo), bf16);
                if (BWD) build_prod_tile<D>(Bs, p.dout, h, p.v2, hk_i, bi, i_base, p.n, k_base, p.nk2, 1.f, bf16);
            }
            bool rvalid[4];
            float lse2[4], dl[4];
#pragma unroll
            for (int ii = 0; ii < 4; ++ii) {
                const int i = i_base + ty + 16 * ii;
                rvalid[ii] = any && i >= ilo && i <= ihi;
                lse2[ii] = 0.f; dl[ii] = 0.f;
                if (BWD && rvalid[ii]) {
                    const int64_t o = ((int64_t)bi * p.hq + h) * p.n + i;
                    lse2[ii] = p.lse[o] * LOG2E;
                    dl[ii] = p.delta[o];
                }
            }
            float u_[4][CPT], w_[4][CPT];      // sums over the window: U (BWD), W (FWD, BWD_K2)
#pragma unroll
            for (int ii = 0; ii < 4; ++ii)
#pragma unroll
                for (int c = 0; c < CPT; ++c) { u_[ii][c] = 0.f; w_[ii][c] = 0.f; }

            int buf = 0;
            for (int j0 = j_lo; j0 <= j_hi; j0 += TILE) {
                float *Ks, *Vs;
                if (C::NBUF == 1 && j0 > j_lo) {
                    __syncthreads();
                    fill_tile<D>(KV, p.k1, bi, hk_i, j0, p.nk1, bf16);
                    fill_tile<D>(KV + TF, p.v1, bi, hk_i, j0, p.nk1, bf16);
                    cp_commit();
                }
                cp_wait<0>();
                __syncthreads();        // this tile has landed, and the other buffer is no longer read
                if (C::NBUF == 2 && j0 + TILE <= j_hi) {
                    float *nx = KV + (buf ^ 1) * 2 * TF;
                    fill_tile<D>(nx, p.k1, bi, hk_i, j0 + TILE, p.nk1, bf16);
                    fill_tile<D>(nx + TF, p.v1, bi, hk_i, j0 + TILE, p.nk1, bf16);
                    cp_commit();
                }
                Ks = KV + (C::NBUF == 2 ? buf : 0) * 2 * TF;
                Vs = Ks + TF;
                buf ^= 1;
                if (!any || ihi + p.off1 < j0 || ilo + p.off1 - p.w1 + 1 > j0 + TILE - 1) continue;

                float s[4][4];
                if (BWD) {
                    // dP waits in the thread's own cells of the G tile: one 4x4 tile less in registers
                    gemm_nt<D>(Bs, Vs, ty, tx, s);
                    __syncwarp();       // the row's last G has been read
#pragma unroll
                    for (int ii = 0; ii < 4; ++ii)
#pragma unroll
                        for (int jj = 0; jj < 4; ++jj) Gs[(ty + 16 * ii) * LP + tx + 16 * jj] = s[ii][jj];
                }
                gemm_nt<D>(As, Ks, ty, tx, s);
                // every cell of the tile valid?
                const bool full = ilo == i_base && ihi == i_base + TILE - 1 && ilo + p.off1 >= j0 + TILE - 1 && ihi + p.off1 - p.w1 < j0;
                const int d0 = i_base + ty + p.off1 - (j0 + tx);         // i + off1 - j of the thread's first cell
                auto ok = [&](int ii, int jj) { return full || (rvalid[ii] && (unsigned)(d0 + 16 * (ii - jj)) < (unsigned)p.w1); };

                if (MODE == MODE_FWD) {
                    // Probabilities against a reference per row that moves only when four of them sum to more than 2^16: the
                    // first tile's maximum mostly serves the whole row, and a sum of P v1 overflows no earlier than 2^22
                    // (64 keys) from the end of the range.
                    float pr[4][4], sum[4];
                    bool exceed = false;
#pragma unroll
                    for (int ii = 0; ii < 4; ++ii) {
                        sum[ii] = 0.f;
#pragma unroll
                        for (int jj = 0; jj < 4; ++jj) {
                            pr[ii][jj] = ok(ii, jj) ? ex2f(s[ii][jj] - ref[ii]) : 0.f;
                            sum[ii] += pr[ii][jj];
                        }
                        exceed |= !(sum[ii] <= 65536.f);
                    }
                    if (__any_sync(0xffffffffu, exceed)) {
#pragma unroll
                        for (int ii = 0; ii < 4; ++ii) {
                            float mx = -CUDART_INF_F;
#pragma unroll
                            for (int jj = 0; jj < 4; ++jj) if (ok(ii, jj)) mx = fmaxf(mx, s[ii][jj]);
                            mx = half_warp_max(mx);
                            // (both branches are uniform over the half-warp that owns the row)
                            if (!(mx > ref[ii])) {
                                // no reference yet, and none here: logits of -inf weigh nothing, and only NaN stays NaN
                                if (ref[ii] > -CUDART_INF_F) continue;
                                sum[ii] = 0.f;
#pragma unroll
                                for (int jj = 0; jj < 4; ++jj) {
                                    pr[ii][jj] = ok(ii, jj) ? ex2f(s[ii][jj]) : 0.f;
                                    sum[ii] += pr[ii][jj];
                                }
                                continue;
                            }
                            const float f = ex2f(ref[ii] - mx);            // 0 on the first hit
                            ref[ii] = mx;
                            l_run[ii] *= f;
                            sum[ii] = 0.f;
#pragma unroll
                            for (int jj = 0; jj < 4; ++jj) {
                                pr[ii][jj] = ok(ii, jj) ? ex2f(s[ii][jj] - mx) : 0.f;
                                sum[ii] += pr[ii][jj];
                            }
#pragma unroll
                            for (int c = 0; c < CPT; ++c) { acc0[ii][c] *= f; w_[ii][c] *= f; }
                        }
                    }
                    __syncwarp();       // the row's last probabilities have been read
#pragma unroll
                    for (int ii = 0; ii < 4; ++ii) {
                        l_run[ii] += sum[ii];
#pragma unroll
                        for (int jj = 0; jj < 4; ++jj) Ps[(ty + 16 * ii) * LP + tx + 16 * jj] = pr[ii][jj];
                    }
                    __syncwarp();
                    gemm_pv<D>(Ps, Vs, ty, tx, w_);
                } else {
#pragma unroll
                    for (int ii = 0; ii < 4; ++ii)
#pragma unroll
                        for (int jj = 0; jj < 4; ++jj) {
                            const int x = (ty + 16 * ii) * LP + tx + 16 * jj;
                            const float pv = ok(ii, jj) ? ex2f(s[ii][jj] - lse2[ii]) : 0.f;
                            Gs[x] = pv * (Gs[x] - dl[ii]);
                            if (MODE == MODE_BWD_K2) Ps[x] = pv;
                        }
                    __syncwarp();
                    gemm_pv<D>(Gs, Ks, ty, tx, u_);
                    if (MODE == MODE_BWD_K2) gemm_pv<D>(Ps, Vs, ty, tx, w_);
                }
            }

            // fold the offset's sums into the rows
#pragma unroll
            for (int ii = 0; ii < 4; ++ii) {
                if (!rvalid[ii]) continue;
                const int i = i_base + ty + 16 * ii, k = k_base + ty + 16 * ii;
#pragma unroll
                for (int u = 0; u < NV; ++u) {
                    float x[VEC], y[VEC];
                    if (MODE == MODE_FWD) load_vec<VEC>(p.v2.p, elem_off(p.v2, bi, k, hk_i) + chan<D>(tx, u), bf16, x);
                    else if (MODE == MODE_BWD_Q) load_vec<VEC>(p.k2.p, elem_off(p.k2, bi, k, hk_i) + chan<D>(tx, u), bf16, x);
                    else {
                        load_vec<VEC>(p.q.p, elem_off(p.q, bi, i, h) + chan<D>(tx, u), bf16, x);
                        load_vec<VEC>(p.dout.p, elem_off(p.dout, bi, i, h) + chan<D>(tx, u), bf16, y);
                    }
#pragma unroll
                    for (int q = 0; q < VEC; ++q) {
                        const int c = u * VEC + q;
                        acc0[ii][c] = fmaf(MODE == MODE_FWD ? w_[ii][c] : u_[ii][c], x[q], acc0[ii][c]);
                        if (MODE == MODE_BWD_K2) acc1[ii][c] = fmaf(w_[ii][c], y[q], acc1[ii][c]);
                    }
                }
            }
        }
    }

    // epilogue: the partial accumulators of all groups meet in shared memory (over the K1/V1 buffers)
    cp_wait<0>();
    __syncthreads();
    cg::cluster_group cl = cg::this_cluster();
    const bool gbf16 = p.grad_bf16 != 0;
    if (MODE == MODE_FWD) {
        put_acc<D>(KV + grp * TF, acc0, ty, tx);
#pragma unroll
        for (int ii = 0; ii < 4; ++ii) {
            const float l = half_warp_sum(l_run[ii]);
            if (tx == 0) {
                stats[(grp * 2) * TILE + ty + 16 * ii] = ref[ii];
                stats[(grp * 2 + 1) * TILE + ty + 16 * ii] = l;
            }
        }
        cl.sync();
        const int rows = TILE / ce;
        for (int idx = threadIdx.x; idx < rows * (D / 4); idx += C::THREADS) {
            const int r = rank * rows + idx / (D / 4), c = (idx % (D / 4)) * 4;
            if (r0 + r >= p.n) continue;
            float M = -CUDART_INF_F, L = 0.f, x[4] = {0.f, 0.f, 0.f, 0.f};
            for (int q = 0; q < ce; ++q)
                for (int g = 0; g < C::NG; ++g) M = fmaxf(M, cl.map_shared_rank(stats, q)[(g * 2) * TILE + r]);
            for (int q = 0; q < ce; ++q)
                for (int g = 0; g < C::NG; ++g) {
                    const float *st = cl.map_shared_rank(stats, q) + g * 2 * TILE;
                    if (!(st[r] > -CUDART_INF_F)) continue;
                    const float f = ex2f(st[r] - M);
                    const float4 v = *reinterpret_cast<const float4 *>(cl.map_shared_rank(KV, q) + g * TF + r * C::LD + c);
                    L = fmaf(st[TILE + r], f, L);
                    x[0] = fmaf(v.x, f, x[0]); x[1] = fmaf(v.y, f, x[1]); x[2] = fmaf(v.z, f, x[2]); x[3] = fmaf(v.w, f, x[3]);
                }
            const float inv = 1.f / L;
#pragma unroll
            for (int z = 0; z < 4; ++z) x[z] *= inv;
            store_vec<4>(p.out.p, elem_off(p.out, bi, r0 + r, h_begin) + c, bf16, x);
            if (c == 0) p.lse[((int64_t)bi * p.hq + h_begin) * p.n + r0 + r] = M * LN2 + __logf(L);
        }
    } else if (MODE == MODE_BWD_Q) {
        put_acc<D>(KV + grp * TF, acc0, ty, tx);
        cl.sync();
        reduce_store<D>(KV, 1, p.dq, bi, h_begin, r0, p.n, p.scale, gbf16);
    } else {
        put_acc<D>(KV + grp * 2 * TF, acc0, ty, tx);
        put_acc<D>(KV + grp * 2 * TF + TF, acc1, ty, tx);
        cl.sync();
        reduce_store<D>(KV, 2, p.dk2, bi, hk_i, r0, p.nk2, p.scale, gbf16);
        reduce_store<D>(KV + TF, 2, p.dv2, bi, hk_i, r0, p.nk2, 1.f, gbf16);
    }
    cl.sync();          // no CTA leaves while its shared memory is read
}

// ---------------------------------------------------------------------------
// First-key-owned tiles: dK1, dV1.  Works on transposed tiles S^T[j][i] so that the accumulators are row-owned.
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void k1_tile(const KernelParams &p, float *smem, int tile, int hk_i, int bi, bool redo) {
    namespace cg = cooperative_groups;
    using C = Cfg<D>;
    constexpr int CPT = C::CPT, TF = C::TF;
    const int grp = threadIdx.x / GROUP, t = threadIdx.x & (GROUP - 1), tx = t & 15, ty = t >> 4;
    float *Ks = smem, *Vs = Ks + TF;
    float *own = smem + 2 * C::NBUF * TF + grp * (2 * TF + 2 * TILE * LP);
    float *As = own, *Bs = As + TF, *Ps = Bs + TF, *Gs = Ps + TILE * LP;

    const int j0 = tile * TILE;
    const bool bf16 = p.in_bf16 != 0;
    int ce, rank;
    cluster_rank(ce, rank);

    fill_tile<D>(Ks, p.k1, bi, hk_i, j0, p.nk1, bf16);
    fill_tile<D>(Vs, p.v1, bi, hk_i, j0, p.nk1, bf16);
    cp_commit();
    cp_wait<0>();
    __syncthreads();

    float dk[4][CPT], dv[4][CPT];
#pragma unroll
    for (int jj = 0; jj < 4; ++jj)
#pragma unroll
        for (int c = 0; c < CPT; ++c) { dk[jj][c] = 0.f; dv[jj][c] = 0.f; }

    const int i_lo = max(0, j0 - p.off1);
    const int i_hi = min(p.n - 1, min(j0 + TILE - 1, p.nk1 - 1) + p.w1 - 1 - p.off1);

    for (int h = hk_i * p.g; h < (hk_i + 1) * p.g; ++h) {
        for (int i0 = i_lo; i0 <= i_hi; i0 += TILE) {
            const int it_hi = min(i0 + TILE - 1, i_hi);
            // column statistics of this query tile
            float lse_c[4], dl_c[4];
#pragma unroll
            for (int ii = 0; ii < 4; ++ii) {
                const int i = i0 + tx + 16 * ii;
                lse_c[ii] = 0.f; dl_c[ii] = 0.f;
                if (i <= it_hi) {
                    const int64_t o = ((int64_t)bi * p.hq + h) * p.n + i;
                    lse_c[ii] = p.lse[o] * LOG2E;
                    dl_c[ii] = p.delta[o];
                }
            }
            for (int e = rank * C::NG + grp; e < p.w2; e += ce * C::NG) {
                const int k_base = i0 + p.off2 - e;
                if (it_hi + p.off2 - e < 0) break;   // no valid second key for any row, nor for larger e
                group_sync(grp);
                build_prod_tile<D>(As, p.q, h, p.k2, hk_i, bi, i0, it_hi + 1, k_base, p.nk2, logit_factor(p.scale, redo), bf16);
                build_prod_tile<D>(Bs, p.dout, h, p.v2, hk_i, bi, i0, it_hi + 1, k_base, p.nk2, 1.f, bf16);
                group_sync(grp);
                float st[4][4];
                gemm_nt<D>(Vs, Bs, ty, tx, st);      // dP^T, which waits in the G tile
                __syncwarp();
#pragma unroll
                for (int jj = 0; jj < 4; ++jj)
#pragma unroll
                    for (int ii = 0; ii < 4; ++ii) Gs[(ty + 16 * jj) * LP + tx + 16 * ii] = st[jj][ii];
                gemm_nt<D>(Ks, As, ty, tx, st);      // st[jj][ii]: row j, column i
                const bool full = it_hi == i0 + TILE - 1 && k_base >= 0 && j0 + TILE - 1 < p.nk1 && i0 + p.off1 >= j0 + TILE - 1 &&
                                  it_hi + p.off1 - p.w1 < j0;
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    const int j = j0 + ty + 16 * jj;
#pragma unroll
                    for (int ii = 0; ii < 4; ++ii) {
                        const int i = i0 + tx + 16 * ii, x = (ty + 16 * jj) * LP + tx + 16 * ii;
                        const bool ok = full || ((i <= it_hi) && (i + p.off2 - e >= 0) && (unsigned)(i + p.off1 - j) < (unsigned)p.w1 && j < p.nk1);
                        const float pv = ok ? ex2f(st[jj][ii] - lse_c[ii]) : 0.f;
                        Gs[x] = pv * (Gs[x] - dl_c[ii]);
                        Ps[x] = pv;
                    }
                }
                __syncwarp();
                gemm_pv<D>(Ps, Bs, ty, tx, dv);
                gemm_pv<D>(Gs, As, ty, tx, dk);
            }
        }
    }

    __syncthreads();
    const bool gbf16 = p.grad_bf16 != 0;
    put_acc<D>(smem + grp * 2 * TF, dk, ty, tx);
    put_acc<D>(smem + grp * 2 * TF + TF, dv, ty, tx);
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    reduce_store<D>(smem, 2, p.dk1, bi, hk_i, j0, p.nk1, redo ? logit_unfactor(p.scale, logit_factor(p.scale, true)) : LN2, gbf16);
    reduce_store<D>(smem + TF, 2, p.dv1, bi, hk_i, j0, p.nk1, 1.f, gbf16);
    cl.sync();
}

// grid: clusters of CTAs along x; forward (tile, query head, batch).  redo: only the tiles whose rows hold LSE_REDO.
template <int D>
__global__ void __launch_bounds__(Cfg<D>::THREADS) fwd_kernel(const KernelParams p, const bool redo) {
    extern __shared__ __align__(16) float smem[];
    const int ce = (int)cooperative_groups::this_cluster().num_blocks();
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (redo && __float_as_uint(p.lse[((int64_t)blockIdx.z * p.hq + blockIdx.y) * p.n + blockIdx.x / ce * TILE]) != LSE_REDO) return;
    row_tile<D, MODE_FWD>(p, smem, blockIdx.x / ce, blockIdx.y, blockIdx.z, redo);
}

// All three gradients: x / cluster size counts the row tiles of dQ, then of dK2/dV2, then of dK1/dV1 (nq, nk2t, nk1t
// of them, already multiplied by their heads), y is the batch.  redo: only the batch elements that it holds a non-zero for, one array
// for dK1/dV1 and one behind it for the others.
struct BwdTiles { int q, k2, k1; };
template <int D>
__global__ void __launch_bounds__(Cfg<D>::THREADS) bwd_kernel(const KernelParams p, const BwdTiles n, const int *redo) {
    extern __shared__ __align__(16) float smem[];
    const int ce = (int)cooperative_groups::this_cluster().num_blocks();
    int x = blockIdx.x / ce;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (redo && !redo[(x >= n.k2 && x < n.k2 + n.k1 ? 0 : p.b) + blockIdx.y]) return;
    // the longest tiles first
    if (x < n.k2) { row_tile<D, MODE_BWD_K2>(p, smem, x / p.hk, x % p.hk, blockIdx.y, redo != nullptr); return; }
    x -= n.k2;
    if (x < n.k1) { k1_tile<D>(p, smem, x / p.hk, x % p.hk, blockIdx.y, redo != nullptr); return; }
    x -= n.k1;
    row_tile<D, MODE_BWD_Q>(p, smem, x / p.hq, x % p.hq, blockIdx.y, redo != nullptr);
}

// D_i = sum_c O_ic dO_ic: D / 8 lanes per (b, i, h) row, eight channels each.  redo (or null): [2][b] flags to clear.
template <int D>
__global__ void __launch_bounds__(256) delta_kernel(const KernelParams p, int *redo) {
    constexpr int LPR = D / 8;
    static_assert(LPR >= 2, "a thread at least for each flag");
    if (redo && (int64_t)blockIdx.x * 256 + threadIdx.x < 2LL * p.b) redo[blockIdx.x * 256 + threadIdx.x] = 0;
    const int64_t rows = (int64_t)p.b * p.n * p.hq;
    const int64_t row = ((int64_t)blockIdx.x * 256 + threadIdx.x) / LPR;
    const int c = (threadIdx.x % LPR) * 8;
    float s = 0.f;
    int h = 0, i = 0, b = 0;
    if (row < rows) {
        h = (int)(row % p.hq);
        i = (int)((row / p.hq) % p.n);
        b = (int)(row / ((int64_t)p.hq * p.n));
        const bool bf16 = p.in_bf16 != 0;
        float a[4], e[4];
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            load_vec<4>(p.out.p, elem_off(p.out, b, i, h) + c + 4 * hf, bf16, a);
            load_vec<4>(p.dout.p, elem_off(p.dout, b, i, h) + c + 4 * hf, bf16, e);
#pragma unroll
            for (int z = 0; z < 4; ++z) s = fmaf(a[z], e[z], s);
        }
    }
#pragma unroll
    for (int o = LPR / 2; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (row < rows && threadIdx.x % LPR == 0) p.delta[((int64_t)b * p.hq + h) * p.n + i] = s;
}

// ------------------------------------------------------------------ host side
// CTAs per row tile: as many as still find an SM of their own, each with two rounds of offsets at least.  A batch
// element's result must not depend on how many ride in the call (bit for bit: callers cut batches into chunks), so
// the rule looks at one element; at large batches a cluster costs the merge of its accumulators, a few per cent.
inline int cluster_size(int64_t tiles_per_element, int w2, int groups, int sms) {
    int ce = 1;
    while (ce < 8 && tiles_per_element * ce * 2 <= sms && w2 >= 2 * ce * groups) ce *= 2;
    return ce;
}

// early: the kernel begins with griddepcontrol.wait, so its blocks may take their places while the kernel before it ends
template <typename K, typename... Args>
inline bool launch_clusters_at(bool early, K kernel, dim3 grid, int threads, size_t smem, int ce, cudaStream_t st, const Args &...args) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return false;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ce; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid; cfg.blockDim = dim3(threads); cfg.dynamicSmemBytes = smem; cfg.stream = st;
    cfg.attrs = attr; cfg.numAttrs = early ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess;
}
template <typename K, typename... Args>
inline bool launch_clusters(K kernel, dim3 grid, int threads, size_t smem, int ce, cudaStream_t st, const Args &...args) {
    return launch_clusters_at(false, kernel, grid, threads, smem, ce, st, args...);
}

template <int D> inline bool launch_delta(const KernelParams &p, cudaStream_t st, int *redo = nullptr) {
    const int64_t threads = (int64_t)p.b * p.n * p.hq * (D / 8);
    delta_kernel<D><<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(p, redo);
    return cudaGetLastError() == cudaSuccess;
}
template <int D> inline bool launch_fwd(const KernelParams &p, int sms, cudaStream_t st, bool redo = false) {
    using C = Cfg<D>;
    const int tiles = (p.n + TILE - 1) / TILE, ce = cluster_size((int64_t)tiles * p.hq, p.w2, C::NG, sms);
    return launch_clusters_at(redo, fwd_kernel<D>, dim3(tiles * ce, p.hq, p.b), C::THREADS, C::smem(false), ce, st, p, redo);
}
// dq / dk2, dv2 / dk1, dv1, those asked for, in one launch
template <int D> inline bool launch_bwd(const KernelParams &p, bool q, bool k2, bool k1, int sms, cudaStream_t st, const int *redo = nullptr) {
    using C = Cfg<D>;
    auto tiles = [](int rows) { return (rows + TILE - 1) / TILE; };
    const BwdTiles n{q ? tiles(p.n) * p.hq : 0, k2 ? tiles(p.nk2) * p.hk : 0, k1 ? tiles(p.nk1) * p.hk : 0};
    // (from the whole backward's tiles, so that a part launched alone gives the same bits)
    const int64_t all = (int64_t)tiles(p.n) * p.hq + (int64_t)(tiles(p.nk2) + tiles(p.nk1)) * p.hk;
    const int ce = cluster_size(all, p.w2, C::NG, sms);
    return launch_clusters_at(redo != nullptr, bwd_kernel<D>, dim3((unsigned)(n.q + n.k2 + n.k1) * ce, p.b), C::THREADS, C::smem(true), ce, st, p, n, redo);
}

}  // namespace simt
}  // namespace sa2
