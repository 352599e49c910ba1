// C ABI of the library (declared in include/sa2.h): argument checks, kernel
// selection and launches.  No torch types, no allocation, no host sync.
#include "sa2.h"
#include "sa2_common.cuh"
#include "sa2_simt.cuh"
#include "sa2_tc.cuh"
#include "sa2_f32.cuh"
#include "sa2_headnorm.cuh"
#include "sa2_rows_linear.cuh"
#include "sa2_step.cuh"
#include <nvtx3/nvToolsExt.h>
#include <type_traits>

namespace sa2 {
namespace nvtx {
// NVTX range around an entry point (header-only NVTX v3: a no-op unless a profiler is attached)
struct Range {
    explicit Range(const char *name) { nvtxRangePushA(name); }
    ~Range() { nvtxRangePop(); }
};
}  // namespace nvtx
}  // namespace sa2

namespace {

using sa2::KernelParams;
using sa2::TensorRef;

inline TensorRef ref(const void *p, const sa2_strides &s) {
    return TensorRef{const_cast<void *>(p), s.batch, s.seq, s.head};
}

inline bool aligned16(const void *p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }
inline bool strides_ok(const sa2_strides &s) { return s.batch % 4 == 0 && s.seq % 4 == 0 && s.head % 4 == 0; }

int check_shape(const sa2_shape &s) {
    if (s.b <= 0 || s.n <= 0 || s.hq <= 0 || s.hk <= 0 || s.w1 <= 0 || s.w2 <= 0) return SA2_ERR_INVALID;
    if (s.off1 < 0 || s.off2 < 0) return SA2_ERR_INVALID;
    if (s.hq % s.hk != 0) return SA2_ERR_INVALID;
    if (s.d != 32 && s.d != 64 && s.d != 128) return SA2_ERR_UNSUPPORTED;
    if (s.dtype != SA2_F32 && s.dtype != SA2_BF16) return SA2_ERR_UNSUPPORTED;
    if (s.kernel != SA2_KERNEL_AUTO && s.kernel != SA2_KERNEL_SIMT && s.kernel != SA2_KERNEL_TCGEN05)
        return SA2_ERR_UNSUPPORTED;
    return SA2_OK;
}

// The shape as the kernels take it.  A row at key position i + off sees at most i + off + 1 <= n + off keys, so a longer
// window selects the same pairs; every rule and loop below may then add tile sizes to w1 and w2 without overflow.
sa2_shape clamped(sa2_shape s) {
    const int64_t nk1 = (int64_t)s.n + s.off1, nk2 = (int64_t)s.n + s.off2;
    if (s.w1 > nk1) s.w1 = (int32_t)nk1;
    if (s.w2 > nk2) s.w2 = (int32_t)nk2;
    return s;
}

void fill_common(KernelParams &p, const sa2_shape &s) {
    p.b = s.b; p.n = s.n; p.hq = s.hq; p.hk = s.hk; p.g = s.hq / s.hk;
    p.w1 = s.w1; p.w2 = s.w2; p.off1 = s.off1; p.off2 = s.off2;
    p.nk1 = s.n + s.off1; p.nk2 = s.n + s.off2;
    p.in_bf16 = (s.dtype == SA2_BF16);
    p.grad_bf16 = 0;
    p.scale = s.scale;
}

inline int launch_status() { return cudaGetLastError() == cudaSuccess ? SA2_OK : SA2_ERR_CUDA; }

template <int D>
int simt_fwd(const KernelParams &p, cudaStream_t st) {
    return sa2::simt::launch_fwd<D>(p, sa2::tc::SM_COUNT, st) ? SA2_OK : SA2_ERR_CUDA;
}

template <int D>
int simt_bwd(const KernelParams &p, cudaStream_t st, int phases = 0) {
    if (phases == 0) phases = SA2_BWD_ROWSUM | SA2_BWD_K1 | SA2_BWD_Q;
    if ((phases & SA2_BWD_ROWSUM) && !sa2::simt::launch_delta<D>(p, st)) return SA2_ERR_CUDA;
    const bool q = phases & SA2_BWD_Q, k1 = phases & SA2_BWD_K1;
    if ((q || k1) && !sa2::simt::launch_bwd<D>(p, q, q, k1, sa2::tc::SM_COUNT, st)) return SA2_ERR_CUDA;
    return SA2_OK;
}

// argument checks shared by sa2_bwd and sa2_bwd_static_scratch
int check_bwd_args(const sa2_bwd_args *a) {
    if (!a) return SA2_ERR_INVALID;
    if (int e = check_shape(a->shape)) return e;
    if (!a->q || !a->k1 || !a->k2 || !a->v1 || !a->v2 || !a->out || !a->dout || !a->lse) return SA2_ERR_INVALID;
    if (!a->dq || !a->dk1 || !a->dk2 || !a->dv1 || !a->dv2) return SA2_ERR_INVALID;
    if (a->grad_dtype != SA2_F32 && a->grad_dtype != SA2_BF16) return SA2_ERR_UNSUPPORTED;
    const void *ptrs[] = {a->q, a->k1, a->k2, a->v1, a->v2, a->out, a->dout, a->dq, a->dk1, a->dk2, a->dv1, a->dv2};
    for (const void *p : ptrs) if (!aligned16(p)) return SA2_ERR_INVALID;
    const sa2_strides *ss[] = {&a->sq, &a->sk1, &a->sk2, &a->sv1, &a->sv2, &a->sout, &a->sdout,
                               &a->sdq, &a->sdk1, &a->sdk2, &a->sdv1, &a->sdv2};
    for (const sa2_strides *s : ss) if (!strides_ok(*s)) return SA2_ERR_INVALID;
    return SA2_OK;
}

void fill_bwd_params(KernelParams &p, const sa2_bwd_args *a, const sa2_shape &s, float *rowsum) {
    fill_common(p, s);
    p.grad_bf16 = (a->grad_dtype == SA2_BF16);
    p.q = ref(a->q, a->sq); p.k1 = ref(a->k1, a->sk1); p.k2 = ref(a->k2, a->sk2);
    p.v1 = ref(a->v1, a->sv1); p.v2 = ref(a->v2, a->sv2);
    p.out = ref(a->out, a->sout); p.dout = ref(a->dout, a->sdout);
    p.dq = ref(a->dq, a->sdq); p.dk1 = ref(a->dk1, a->sdk1); p.dk2 = ref(a->dk2, a->sdk2);
    p.dv1 = ref(a->dv1, a->sdv1); p.dv2 = ref(a->dv2, a->sdv2);
    p.lse = const_cast<float *>(a->lse);
    p.delta = rowsum;
}

// One block of one warp waits on a barrier that nobody arrives on, with the given limit: the self-test of
// the bounded waits.  The wait runs out, the block records ERR_SELFTEST and leaves through the normal path.
__global__ void selftest_wait_kernel(long long limit_cycles, int *status) {
    __shared__ uint64_t bar;
    __shared__ int abort_flag;
    if (threadIdx.x == 0) {
        sa2::sm100::mbar_init(&bar, 1);
        abort_flag = 0;
        sa2::sm100::fence_barrier_init();
    }
    __syncthreads();
    const bool ok = sa2::sm100::mbar_wait(&bar, 0, &abort_flag, 32, -1, limit_cycles);
    if (!ok && threadIdx.x == 0) atomicOr(status, SA2_SELFTEST_WAIT_BIT);
}

}  // namespace

extern "C" {

int sa2_version(void) { return 100; }

int sa2_selftest_wait(long long limit_cycles, void *stream) {
    if (limit_cycles <= 0 || limit_cycles > 2000000000LL) return SA2_ERR_INVALID;
    int *word = sa2::tc::status_word();
    if (!word) return SA2_ERR_CUDA;
    selftest_wait_kernel<<<1, 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(limit_cycles, word);
    return launch_status();
}

#ifdef SA2_PROF
// diagnostic builds only (-DSA2_PROF=<CTA index>): read and clear the wait-accounting table
int sa2_prof_read(unsigned long long *host, int n) {
    if (cudaMemcpyFromSymbol(host, sa2::sm100::g_prof, sizeof(unsigned long long) * n) != cudaSuccess) return -1;
    static unsigned long long zeros[512] = {0};
    return cudaMemcpyToSymbol(sa2::sm100::g_prof, zeros, sizeof(unsigned long long) * n) == cudaSuccess ? 0 : -1;
}
#endif

int sa2_device_status(int reset) {
    int *word = sa2::tc::status_word();
    if (!word) return -1;
    int v = 0;
    if (cudaMemcpy(&v, word, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    if (reset && v != 0) {
        const int zero = 0;
        if (cudaMemcpy(word, &zero, sizeof(int), cudaMemcpyHostToDevice) != cudaSuccess) return -1;
    }
    return v;
}

int sa2_check_device(int reset) {
    const int v = sa2_device_status(reset);
    if (v < 0) return SA2_ERR_CUDA;
    return v == 0 ? SA2_OK : SA2_ERR_DEVICE;
}

const char *sa2_strerror(int status) {
    switch (status) {
        case SA2_OK: return "ok";
        case SA2_ERR_INVALID: return "invalid argument (null pointer, bad size, hq % hk != 0, misaligned pointer or stride)";
        case SA2_ERR_UNSUPPORTED: return "unsupported configuration (head dim must be 32, 64 or 128; dtype fp32 or bf16; "
                                         "the tcgen05 kernels need bf16)";
        case SA2_ERR_WORKSPACE: return "workspace missing, misaligned or smaller than sa2_bwd_workspace_bytes()";
        case SA2_ERR_CUDA: return "a CUDA call failed";
        case SA2_ERR_DEVICE: return "a kernel gave up on a bounded wait; the rows it owned hold NaN";
        case SA2_ERR_TOO_LARGE: return "problem too large for the library's built-in scratch: b * hq * n exceeds "
                                       "SA2_STATIC_SCRATCH_ROWS (use sa2_bwd with a caller-provided workspace)";
        default: return "unknown status";
    }
}

int sa2_kernel_launches(const sa2_shape *shape, int backward) {
    if (!shape || check_shape(*shape) != SA2_OK) return -1;
    const sa2_shape s = clamped(*shape);
    const bool tc_ok = backward ? sa2::tc::bwd_supported(s) : sa2::tc::fwd_supported(s);
    if (s.kernel == SA2_KERNEL_TCGEN05 && !tc_ok) return -1;
    if (tc_ok && s.kernel != SA2_KERNEL_SIMT && !(backward && !sa2::tc::bwd_scale_ok(s)))
        return sa2::tc::launches(s, backward != 0, {shape->w2, shape->b});
    if (sa2::f32::supported(s)) return backward ? sa2::f32::bwd_launches(s, shape->b, sa2::tc::SM_COUNT) : 2;
    return backward ? 2 : 1;   // SIMT: row sums + all gradients
}

size_t sa2_bwd_workspace_bytes_part(const sa2_shape *shape, int32_t whole_b) {
    if (!shape || check_shape(*shape) != SA2_OK || whole_b < shape->b) return 0;
    const sa2_shape s = clamped(*shape);
    size_t delta = (size_t)s.b * s.hq * s.n * sizeof(float);
    delta = (delta + 255) & ~(size_t)255;
    if (sa2::f32::supported(s)) return delta + sa2::f32::bwd_workspace_bytes(s, whole_b, sa2::tc::SM_COUNT);
    return delta + sa2::tc::bwd_extra_workspace_bytes(s, {shape->w2, whole_b});
}

size_t sa2_bwd_workspace_bytes(const sa2_shape *shape) { return shape ? sa2_bwd_workspace_bytes_part(shape, shape->b) : 0; }

int sa2_fwd(const sa2_fwd_args *a) {
    sa2::nvtx::Range range("sa2_fwd");
    if (!a) return SA2_ERR_INVALID;
    if (int e = check_shape(a->shape)) return e;
    if (!a->q || !a->k1 || !a->k2 || !a->v1 || !a->v2 || !a->out || !a->lse) return SA2_ERR_INVALID;
    const void *ptrs[] = {a->q, a->k1, a->k2, a->v1, a->v2, a->out};
    for (const void *p : ptrs) if (!aligned16(p)) return SA2_ERR_INVALID;
    const sa2_strides *ss[] = {&a->sq, &a->sk1, &a->sk2, &a->sv1, &a->sv2, &a->sout};
    for (const sa2_strides *s : ss) if (!strides_ok(*s)) return SA2_ERR_INVALID;

    const sa2_shape s = clamped(a->shape);
    KernelParams p{};
    fill_common(p, s);
    p.q = ref(a->q, a->sq); p.k1 = ref(a->k1, a->sk1); p.k2 = ref(a->k2, a->sk2);
    p.v1 = ref(a->v1, a->sv1); p.v2 = ref(a->v2, a->sv2); p.out = ref(a->out, a->sout);
    p.lse = a->lse;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(a->stream);

    const bool tc_ok = sa2::tc::fwd_supported(s) && sa2::tc::fwd_addressable(p);
    if (s.kernel == SA2_KERNEL_TCGEN05 && !tc_ok) return SA2_ERR_UNSUPPORTED;
    if (tc_ok && s.kernel != SA2_KERNEL_SIMT) return sa2::tc::fwd(p, s, sa2::tc::fwd_split(a->shape), st);

    if (sa2::f32::supported(s)) {
        int *status = sa2::tc::status_word();
        if (!status) return SA2_ERR_CUDA;
        return s.d == 32 ? sa2::f32::fwd<32>(p, status, sa2::tc::SM_COUNT, st) : sa2::f32::fwd<64>(p, status, sa2::tc::SM_COUNT, st);
    }

    switch (s.d) {
        case 32: return simt_fwd<32>(p, st);
        case 64: return simt_fwd<64>(p, st);
        default: return simt_fwd<128>(p, st);
    }
}

int sa2_bwd(const sa2_bwd_args *a) { return sa2_bwd_part(a, a ? a->shape.b : 0); }

int sa2_bwd_part(const sa2_bwd_args *a, int32_t whole_b) {
    sa2::nvtx::Range range("sa2_bwd");
    if (int e = check_bwd_args(a)) return e;
    if (whole_b < a->shape.b) return SA2_ERR_INVALID;
    if (a->phases < 0 || a->phases > (SA2_BWD_ROWSUM | SA2_BWD_K1 | SA2_BWD_Q)) return SA2_ERR_INVALID;
    const size_t need = sa2_bwd_workspace_bytes_part(&a->shape, whole_b);
    if (!a->workspace || a->workspace_bytes < need || (reinterpret_cast<uintptr_t>(a->workspace) & 255u))
        return SA2_ERR_WORKSPACE;

    const sa2_shape s = clamped(a->shape);
    KernelParams p{};
    fill_bwd_params(p, a, s, reinterpret_cast<float *>(a->workspace));
    cudaStream_t st = reinterpret_cast<cudaStream_t>(a->stream);

    const bool tc_ok = sa2::tc::bwd_supported(s) && sa2::tc::bwd_addressable(p);
    if (s.kernel == SA2_KERNEL_TCGEN05 && !tc_ok) return SA2_ERR_UNSUPPORTED;
    // (fp32 gradients at head dim 32 show the last bits, which AUTO leaves to the fp32 kernels)
    const bool exact = s.kernel == SA2_KERNEL_AUTO && s.d == 32 && a->grad_dtype == SA2_F32;
    size_t delta = (size_t)s.b * s.hq * s.n * sizeof(float);
    delta = (delta + 255) & ~(size_t)255;
    if (tc_ok && s.kernel != SA2_KERNEL_SIMT && !exact && sa2::tc::bwd_scale_ok(s)) {
        return sa2::tc::bwd(p, s, {a->shape.w2, whole_b}, reinterpret_cast<char *>(a->workspace) + delta, st, a->phases);
    }

    if (sa2::f32::supported(s)) {
        const sa2::f32::Plan plan = sa2::f32::plan(s, whole_b, sa2::tc::SM_COUNT);
        int *status = sa2::tc::status_word();
        if (!status) return SA2_ERR_CUDA;
        char *extra = reinterpret_cast<char *>(a->workspace) + delta;
        if (plan.tc) return s.d == 32 ? sa2::f32::bwd<32>(p, plan, extra, status, sa2::tc::SM_COUNT, st, a->phases)
                                    : sa2::f32::bwd<64>(p, plan, extra, status, sa2::tc::SM_COUNT, st, a->phases);
    }

    switch (s.d) {
        case 32: return simt_bwd<32>(p, st, a->phases);
        case 64: return simt_bwd<64>(p, st, a->phases);
        default: return simt_bwd<128>(p, st, a->phases);
    }
}

// ---------------------------------------------------------------------------
// Backward without caller-provided scratch.
//
// Some hosts of this library cannot hand it a workspace: an inference or
// training engine that claimed all device memory for its own pools at start-up,
// a plug-in that is only allowed to launch kernels, a latency-critical loop in
// which every allocator call is forbidden.  For them the row sums
// D_i = sum_c O_ic dO_ic live in the fixed device array below instead.  The
// array is part of the library image: every GPU that loads the library keeps
// SA2_STATIC_SCRATCH_ROWS * 4 bytes (1 MiB) for it until the process exits.
// ---------------------------------------------------------------------------
static __device__ __align__(256) float g_static_rowsum[SA2_STATIC_SCRATCH_ROWS];

namespace {

// Device address of g_static_rowsum on the current device.  In host code the
// array's name is only a handle, never a device pointer, so the address is
// asked for once per device (with that device current) and remembered.
float *static_rowsum_ptr() {
    static float *ptrs[64] = {nullptr};
    int dev = -1;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    float *p = ptrs[dev];
    if (!p) {
        void *addr = nullptr;
        if (cudaGetSymbolAddress(&addr, g_static_rowsum) != cudaSuccess || !addr) return nullptr;
        p = reinterpret_cast<float *>(addr);
        ptrs[dev] = p;      // racing first calls store the same value
    }
    return p;
}

}  // namespace

int sa2_bwd_static_scratch(const sa2_bwd_args *a) {
    sa2::nvtx::Range range("sa2_bwd_static_scratch");
    if (int e = check_bwd_args(a)) return e;
    // only the fp32 kernels get by with the row sums alone
    if (a->shape.kernel == SA2_KERNEL_TCGEN05) return SA2_ERR_UNSUPPORTED;
    const long long rows = (long long)a->shape.b * a->shape.hq * a->shape.n;
    if (rows > (long long)SA2_STATIC_SCRATCH_ROWS) return SA2_ERR_TOO_LARGE;

    float *rowsum = static_rowsum_ptr();
    if (!rowsum) return SA2_ERR_CUDA;

    const sa2_shape s = clamped(a->shape);
    KernelParams p{};
    fill_bwd_params(p, a, s, rowsum);    // every entry the kernels read is rewritten first: nothing has to start at zero
    cudaStream_t st = reinterpret_cast<cudaStream_t>(a->stream);
    switch (s.d) {
        case 32: return simt_bwd<32>(p, st);
        case 64: return simt_bwd<64>(p, st);
        default: return simt_bwd<128>(p, st);
    }
}

}  // extern "C"

// ---------------------------------------------------------------- per-head RMSNorm
namespace {

int headnorm_grid(int64_t rows) {
    const int64_t want = (rows + sa2::headnorm::WARPS - 1) / sa2::headnorm::WARPS;
    return (int)(want < 592 ? (want > 0 ? want : 1) : 592);          // 4 CTAs per SM
}

int headnorm_check(const sa2_headnorm_args *a, bool backward) {
    if (!a || !a->x || !a->weight || !a->y || !a->rstd || a->rows <= 0 || a->channels <= 0) return SA2_ERR_INVALID;
    if (a->d != 32 && a->d != 64 && a->d != 128 && a->d != 256 && a->d != 512) return SA2_ERR_UNSUPPORTED;
    if (a->channels % a->d != 0) return SA2_ERR_INVALID;
    if ((a->x_dtype != SA2_F32 && a->x_dtype != SA2_BF16) || (a->y_dtype != SA2_F32 && a->y_dtype != SA2_BF16)) return SA2_ERR_UNSUPPORTED;
    if (a->x_stride < a->channels || a->y_stride < a->channels) return SA2_ERR_INVALID;
    if (backward) {
        if (!a->dy || !a->dweight || a->dy_stride < a->channels) return SA2_ERR_INVALID;
        if (!a->partial || a->partial_bytes < sa2_headnorm_partial_bytes(a->rows, a->channels)) return SA2_ERR_WORKSPACE;
    }
    return SA2_OK;
}

using sa2::headnorm::Gains;
using sa2::headnorm::GainGrads;

inline int rows_aligned(const void *p, int64_t stride, int dtype) {
    return aligned16(p) && stride % (dtype == SA2_BF16 ? 8 : 4) == 0;
}

template <typename TX, typename TY, int D>
int headnorm_run(const sa2::headnorm::Params &P, bool backward, float *dtable, const GainGrads &grads, cudaStream_t st) {
    using namespace sa2::headnorm;
    const int segs = (P.channels + Seg<D>::CH - 1) / Seg<D>::CH;
    if (!backward) {
        const int64_t blocks = (P.rows * segs + 7) / 8;
        fwd_kernel<TX, TY, D><<<(unsigned)(blocks < 148 * 64 ? blocks : 148 * 64), 256, 0, st>>>(P);
        return launch_status();
    }
    const int grid = headnorm_grid(P.rows);
    const int rpc = segs >= 8 ? 1 : 8 / segs;
    const size_t smem = (size_t)(rpc - 1) * P.channels * sizeof(float);
    bwd_kernel<TX, TY, D><<<grid, 32 * segs * rpc, smem, st>>>(P);        // at most 7/8 * 8 warps * 2 KB of shared memory
    if (int e = launch_status()) return e;
    const dim3 rgrid = dtable ? dim3((P.channels + 31) / 32) : dim3(D / 32, 5);
    dgain_reduce_kernel<<<rgrid, 1024, 0, st>>>(P.partial, dtable, grads, P.gains, grid, P.channels, D);
    return launch_status();
}

template <typename TX, typename TY>
int headnorm_launch(const sa2::headnorm::Params &P, int d, bool backward, float *dtable, const GainGrads &grads, cudaStream_t st) {
    switch (d) {
        case 32: return headnorm_run<TX, TY, 32>(P, backward, dtable, grads, st);
        case 64: return headnorm_run<TX, TY, 64>(P, backward, dtable, grads, st);
        case 128: return headnorm_run<TX, TY, 128>(P, backward, dtable, grads, st);
        case 256: return headnorm_run<TX, TY, 256>(P, backward, dtable, grads, st);
        default: return headnorm_run<TX, TY, 512>(P, backward, dtable, grads, st);
    }
}

int headnorm_types(const sa2::headnorm::Params &P, int d, int x_dtype, int y_dtype, bool backward, float *dtable,
                   const GainGrads &grads, cudaStream_t st) {
    // a CTA of the backward spans a row: 32 warps of 256 channels
    if (backward && P.channels > 6400) return SA2_ERR_UNSUPPORTED;
    const bool xb = x_dtype == SA2_BF16, yb = y_dtype == SA2_BF16;
    if (xb && yb) return headnorm_launch<__nv_bfloat16, __nv_bfloat16>(P, d, backward, dtable, grads, st);
    if (xb) return headnorm_launch<__nv_bfloat16, float>(P, d, backward, dtable, grads, st);
    if (yb) return headnorm_launch<float, __nv_bfloat16>(P, d, backward, dtable, grads, st);
    return headnorm_launch<float, float>(P, d, backward, dtable, grads, st);
}

int headnorm_dispatch(const sa2_headnorm_args *a, bool backward) {
    const int rc = headnorm_check(a, backward);
    if (rc != SA2_OK) return rc;
    sa2::headnorm::Params P{};
    P.x = a->x; P.dy = a->dy; P.y = a->y; P.rstd = a->rstd;
    P.gains.table = a->weight;
    P.gains.al = aligned16(a->weight);
    P.partial = reinterpret_cast<float *>(a->partial);
    P.partial_al = aligned16(a->partial);
    P.rows = a->rows; P.x_stride = a->x_stride; P.y_stride = a->y_stride; P.dy_stride = a->dy_stride;
    P.channels = a->channels; P.eps = a->eps;
    P.x_al = rows_aligned(a->x, a->x_stride, a->x_dtype);
    P.y_al = rows_aligned(a->y, a->y_stride, backward ? a->x_dtype : a->y_dtype);
    P.dy_al = backward && rows_aligned(a->dy, a->dy_stride, a->y_dtype);
    return headnorm_types(P, a->d, a->x_dtype, a->y_dtype, backward, a->dweight, GainGrads{}, reinterpret_cast<cudaStream_t>(a->stream));
}

int qkvnorm_fill(const sa2_qkvnorm_args *a, bool backward, sa2::headnorm::Params &P, GainGrads &grads) {
    if (!a || !a->x || !a->y || a->rows <= 0 || a->hq <= 0 || a->hk < 0) return SA2_ERR_INVALID;
    const bool whole_row = a->hk == 0 && a->hq == 1 && !backward;      // the module's prenorm / postnorm
    if (a->hk == 0 && !whole_row) return SA2_ERR_INVALID;
    if (a->d != 32 && a->d != 64 && a->d != 128 && !(whole_row && (a->d == 256 || a->d == 512))) return SA2_ERR_UNSUPPORTED;
    for (int dt : {a->x_dtype, a->y_dtype, a->gain_dtype})
        if (dt != SA2_F32 && dt != SA2_BF16) return SA2_ERR_UNSUPPORTED;
    const int64_t channels = (int64_t)a->d * (a->hq + 4LL * a->hk);
    if (channels > 1 << 20 || a->x_stride < channels) return SA2_ERR_INVALID;
    P = sa2::headnorm::Params{};
    grads = GainGrads{};
    for (int v = 0; v < (whole_row ? 1 : 5); ++v) {
        if (!a->gain[v] || !aligned16(a->gain[v])) return SA2_ERR_INVALID;
        P.gains.p[v] = a->gain[v];
        grads.p[v] = a->dgain[v];
        if (backward && !a->dgain[v]) return SA2_ERR_INVALID;
    }
    P.gains.bf16 = grads.bf16 = a->gain_dtype == SA2_BF16;
    P.gains.hq = a->hq; P.gains.hk = a->hk;
    P.x = a->x; P.dy = a->dy; P.y = a->y; P.rstd = a->rstd;
    P.partial = reinterpret_cast<float *>(a->partial);
    P.partial_al = aligned16(a->partial);
    P.rows = a->rows; P.x_stride = a->x_stride; P.y_stride = a->y_stride; P.dy_stride = a->dy_stride;
    P.channels = (int)channels; P.eps = a->eps;
    P.x_al = rows_aligned(a->x, a->x_stride, a->x_dtype);
    P.y_al = rows_aligned(a->y, a->y_stride, backward ? a->x_dtype : a->y_dtype);
    P.dy_al = backward && rows_aligned(a->dy, a->dy_stride, a->y_dtype);
    return SA2_OK;
}

int qkvnorm_dispatch(const sa2_qkvnorm_args *a, bool backward) {
    sa2::headnorm::Params P;
    GainGrads grads;
    if (int e = qkvnorm_fill(a, backward, P, grads)) return e;
    if (a->y_stride < P.channels) return SA2_ERR_INVALID;
    if (backward) {
        if (!a->rstd || !a->dy || a->dy_stride < P.channels) return SA2_ERR_INVALID;
        if (!a->partial || a->partial_bytes < sa2_headnorm_partial_bytes(a->rows, P.channels)) return SA2_ERR_WORKSPACE;
    }
    return headnorm_types(P, a->d, a->x_dtype, a->y_dtype, backward, nullptr, grads, reinterpret_cast<cudaStream_t>(a->stream));
}

template <typename T>
int append_launch(const sa2::headnorm::AppendParams &A, int d, cudaStream_t st) {
    using namespace sa2::headnorm;
    const int64_t want = (A.copy_items + 1023) / 1024;           // four pieces per thread
    const unsigned grid = (unsigned)((A.norm_items + 7) / 8 + (want < 148 * 8 ? want : 148 * 8));
    if (d == 32) append_kernel<T, 32><<<grid, 256, 0, st>>>(A);
    else if (d == 64) append_kernel<T, 64><<<grid, 256, 0, st>>>(A);
    else append_kernel<T, 128><<<grid, 256, 0, st>>>(A);
    return launch_status();
}

int rows_linear_run(const void *x, const void *gain, int gain_dtype, float eps, const void *w, void *y, int rows, int k, int outs, void *stream) {
    using namespace sa2::rows_linear;
    if (!x || !w || !y || rows <= 0 || k <= 0 || outs <= 0 || !aligned16(x) || !aligned16(w) || !aligned16(y) || (gain && !aligned16(gain))) return SA2_ERR_INVALID;
    if (rows > MAX_NORM_ROWS || k % 32 || outs % OUTS) return SA2_ERR_UNSUPPORTED;
    auto pick = [&](auto normed) {
        constexpr bool N = decltype(normed)::value;
        return rows <= 8 ? kernel<1, N> : rows <= 16 ? kernel<2, N> : rows <= 32 ? kernel<4, N> : kernel<8, N>;
    };
    auto run = gain ? pick(std::true_type{}) : pick(std::false_type{});
    run<<<outs / OUTS, WARPS * 32, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const __nv_bfloat16 *>(x), reinterpret_cast<const __nv_bfloat16 *>(w), reinterpret_cast<__nv_bfloat16 *>(y), rows, k, outs,
        Norm{gain, gain_dtype == SA2_BF16, eps});
    return launch_status();
}

}  // namespace

extern "C" {

size_t sa2_headnorm_partial_bytes(int64_t rows, int32_t channels) {
    if (rows <= 0 || channels <= 0) return 0;
    return (size_t)headnorm_grid(rows) * (size_t)channels * sizeof(float);
}
int sa2_headnorm_fwd(const sa2_headnorm_args *a) {
    sa2::nvtx::Range range("sa2_headnorm_fwd");
    return headnorm_dispatch(a, false);
}
int sa2_headnorm_bwd(const sa2_headnorm_args *a) {
    sa2::nvtx::Range range("sa2_headnorm_bwd");
    return headnorm_dispatch(a, true);
}

int sa2_qkvnorm_fwd(const sa2_qkvnorm_args *a) {
    sa2::nvtx::Range range("sa2_qkvnorm_fwd");
    return qkvnorm_dispatch(a, false);
}
int sa2_qkvnorm_bwd(const sa2_qkvnorm_args *a) {
    sa2::nvtx::Range range("sa2_qkvnorm_bwd");
    return qkvnorm_dispatch(a, true);
}
int sa2_qkv_append(const sa2_qkvnorm_args *a, const sa2_append_set *sets, int32_t b, int32_t n) {
    sa2::nvtx::Range range("sa2_qkv_append");
    sa2::headnorm::AppendParams A{};
    GainGrads grads;
    if (int e = qkvnorm_fill(a, false, A.norm, grads)) return e;
    if (!sets || a->hk == 0 || b <= 0 || n <= 0 || a->rows != (int64_t)b * n || a->x_dtype != a->y_dtype || !aligned16(a->y)) return SA2_ERR_INVALID;
    const int piece = a->x_dtype == SA2_BF16 ? 8 : 4;
    const int64_t segs = (A.norm.channels + 255) / 256, items = a->rows * segs;
    if (items > 1 << 28) return SA2_ERR_UNSUPPORTED;
    A.b = b; A.n = n; A.hq = a->hq; A.hk = a->hk;
    A.norm_items = (int)items;
    for (int s = 0; s < 4; ++s) {
        const sa2_append_set &t = sets[s];
        if (t.keep < 0 || !t.dst || !aligned16(t.dst)) return SA2_ERR_INVALID;
        if (t.keep > 0 && (!t.cache || !aligned16(t.cache) || t.strides.batch % piece || t.strides.seq % piece || t.strides.head % piece))
            return SA2_ERR_INVALID;
        A.set[s] = sa2::headnorm::AppendSet{t.cache, t.strides.batch, t.strides.seq, t.strides.head, t.dst, t.keep};
        A.copy_items += (int64_t)b * t.keep * a->hk * (a->d / piece);
    }
    cudaStream_t st = reinterpret_cast<cudaStream_t>(a->stream);
    return a->x_dtype == SA2_BF16 ? append_launch<__nv_bfloat16>(A, a->d, st) : append_launch<float>(A, a->d, st);
}

int sa2_rows_linear(const void *x, const void *w, void *y, int32_t rows, int32_t k, int32_t outs, void *stream) {
    sa2::nvtx::Range range("sa2_rows_linear");
    if (rows > sa2::rows_linear::MAX_ROWS) return x && w && y && k > 0 && outs > 0 ? SA2_ERR_UNSUPPORTED : SA2_ERR_INVALID;
    return rows_linear_run(x, nullptr, 0, 0.f, w, y, rows, k, outs, stream);
}

int sa2_norm_linear(const void *x, const void *gain, int32_t gain_dtype, float eps, const void *w, void *y, int32_t rows, int32_t k, int32_t outs, void *stream) {
    sa2::nvtx::Range range("sa2_norm_linear");
    if (gain && gain_dtype != SA2_F32 && gain_dtype != SA2_BF16) return SA2_ERR_UNSUPPORTED;
    return rows_linear_run(x, gain, gain_dtype, eps, w, y, rows, k, outs, stream);
}

int sa2_step_attn(const sa2_qkvnorm_args *a, const sa2_append_set *sets, void *out, int32_t b, int32_t w1, int32_t w2, float scale) {
    sa2::nvtx::Range range("sa2_step_attn");
    if (!a || !a->x || !sets || !out || !aligned16(out) || b <= 0 || a->rows != b || a->hq <= 0 || a->hk <= 0 || a->hq % a->hk || w1 <= 0 || w2 <= 0)
        return SA2_ERR_INVALID;
    if ((a->d != 64 && a->d != 128) || a->x_dtype != SA2_BF16 || (a->gain_dtype != SA2_F32 && a->gain_dtype != SA2_BF16) || w2 > sa2::step::MAX_W2)
        return SA2_ERR_UNSUPPORTED;
    if (a->x_stride < (int64_t)a->d * (a->hq + 4LL * a->hk) || !rows_aligned(a->x, a->x_stride, SA2_BF16)) return SA2_ERR_INVALID;
    sa2::step::Params P{};
    for (int v = 0; v < 5; ++v) {
        if (!a->gain[v] || !aligned16(a->gain[v])) return SA2_ERR_INVALID;
        P.gains.p[v] = a->gain[v];
    }
    P.gains.bf16 = a->gain_dtype == SA2_BF16;
    P.gains.hq = a->hq; P.gains.hk = a->hk;
    P.proj = reinterpret_cast<const __nv_bfloat16 *>(a->x);
    P.stride = a->x_stride; P.eps = a->eps; P.c = scale * 1.4426950408889634f;
    for (int s = 0; s < 4; ++s) {
        const sa2_append_set &t = sets[s];
        const int w = s & 1 ? w2 : w1, rows = t.keep + 1 < w ? t.keep + 1 : w - 1;
        if (t.keep < 0 || t.keep != sets[s & 1].keep || (rows > 0 && (!t.dst || !aligned16(t.dst)))) return SA2_ERR_INVALID;
        if (t.keep > 0 && (!t.cache || !aligned16(t.cache) || t.strides.batch % 8 || t.strides.seq % 8 || t.strides.head % 8)) return SA2_ERR_INVALID;
        P.set[s] = sa2::step::Set{reinterpret_cast<const __nv_bfloat16 *>(t.cache), t.strides.batch, t.strides.seq, t.strides.head,
                                  reinterpret_cast<__nv_bfloat16 *>(t.dst), t.keep, rows};
    }
    P.out = reinterpret_cast<__nv_bfloat16 *>(out);
    P.hq = a->hq; P.hk = a->hk; P.g = a->hq / a->hk; P.w1 = w1; P.w2 = w2;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(a->stream);
    const int rc = a->d == 64 ? sa2::step::launch<64>(P, b, sa2::tc::SM_COUNT, st) : sa2::step::launch<128>(P, b, sa2::tc::SM_COUNT, st);
    return rc < 0 ? SA2_ERR_UNSUPPORTED : rc == 0 ? SA2_OK : SA2_ERR_CUDA;
}

}  // extern "C"
