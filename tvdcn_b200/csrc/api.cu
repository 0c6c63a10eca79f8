// C ABI (include/tvdcn_b200.h): validation, engine choice, workspace layout, kernel sequencing.
#include <cstdlib>
#include <atomic>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/tvdcn_b200.h"
#include "kernels.h"
#include "plan.h"
#include "sm100_ptx.cuh"

namespace tvdcn_b200 {

static std::atomic<uint64_t> g_launches{0};
void count_launch(int n) { g_launches.fetch_add((uint64_t)n, std::memory_order_relaxed); }

// ---- optional per-kernel timing (CUDA events on the launching stream) -----------------------------
struct TimedLaunch {
    const char *name;
    cudaEvent_t start, stop;
};
static std::atomic<int> g_timing{0};
static std::mutex g_timing_mu;
static std::vector<TimedLaunch> g_timed;

LaunchScope::LaunchScope(const char *name, cudaStream_t stream) : name_(name), stream_(stream) {
    count_launch();
    if (g_timing.load(std::memory_order_relaxed)) {
        if (cudaEventCreate(&start_) == cudaSuccess) cudaEventRecord(start_, stream_);
        else start_ = nullptr;
    }
}

LaunchScope::~LaunchScope() {
    if (start_ == nullptr) return;
    cudaEvent_t stop;
    if (cudaEventCreate(&stop) != cudaSuccess) { cudaEventDestroy(start_); return; }
    cudaEventRecord(stop, stream_);
    std::lock_guard<std::mutex> lk(g_timing_mu);
    g_timed.push_back({name_, start_, stop});
}

static thread_local char g_err[512] = "";

int fail(int code, const char *fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
    return code;
}

int cuda_fail(cudaError_t e, const char *what) {
    return fail(TVDCN_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
}

static int64_t prod(const int64_t *v, int n) {
    int64_t r = 1;
    for (int i = 0; i < n; ++i) r *= v[i];
    return r;
}

int check_problem(const tvdcn_problem *p) {
    if (p == nullptr) return fail(TVDCN_ERR_INVALID, "problem is NULL");
    if (p->dim < 1 || p->dim > 3) return fail(TVDCN_ERR_INVALID, "dim must be 1, 2 or 3 (got %d)", p->dim);
    if (p->dtype < TVDCN_F32 || p->dtype > TVDCN_BF16) return fail(TVDCN_ERR_INVALID, "unknown dtype %d", p->dtype);
    if ((p->flags & ~TVDCN_FLAG_REUSE_STAGED_INPUT) != 0) return fail(TVDCN_ERR_INVALID, "unknown flags 0x%x", p->flags);
    const bool aux_ok = p->aux_dtype == p->dtype ||
                        (p->aux_dtype == TVDCN_F32 && (p->dtype == TVDCN_F16 || p->dtype == TVDCN_BF16));
    if (!aux_ok)
        return fail(TVDCN_ERR_INVALID, "aux_dtype must equal dtype, or be f32 beside a 16-bit dtype (got %d / %d)",
                    p->dtype, p->aux_dtype);
    if (p->batch < 0 || p->in_channels <= 0 || p->out_channels <= 0)
        return fail(TVDCN_ERR_INVALID, "batch / channel counts must be positive");
    if (p->groups <= 0 || p->in_channels % p->groups != 0 || p->out_channels % p->groups != 0)
        return fail(TVDCN_ERR_INVALID, "in_channels (%lld) and out_channels (%lld) must be divisible by groups (%d)",
                    (long long)p->in_channels, (long long)p->out_channels, p->groups);
    const int64_t cs = p->transposed ? p->out_channels : p->in_channels;
    if (p->offset_groups < 0 || (p->offset_groups > 0 && cs % p->offset_groups != 0))
        return fail(TVDCN_ERR_INVALID, "sampled channels (%lld) must be divisible by offset_groups (%d)",
                    (long long)cs, p->offset_groups);
    if (p->mask_groups < 0 || (p->mask_groups > 0 && cs % p->mask_groups != 0))
        return fail(TVDCN_ERR_INVALID, "sampled channels (%lld) must be divisible by mask_groups (%d)",
                    (long long)cs, p->mask_groups);
    for (int a = 0; a < p->dim; ++a) {
        if (p->kernel[a] <= 0 || p->stride[a] <= 0 || p->dilation[a] <= 0 || p->padding[a] < 0 ||
            p->in_size[a] <= 0)
            return fail(TVDCN_ERR_INVALID, "axis %d: kernel %d stride %d padding %d dilation %d in_size %lld", a,
                        p->kernel[a], p->stride[a], p->padding[a], p->dilation[a], (long long)p->in_size[a]);
        if (p->transposed && p->output_padding[a] < 0)
            return fail(TVDCN_ERR_INVALID, "axis %d: negative output_padding", a);
    }
    return TVDCN_OK;
}

static int check_sizes(const tvdcn_problem *p) {
    for (int a = 0; a < p->dim; ++a)
        if (p->out_size[a] <= 0)
            return fail(TVDCN_ERR_INVALID, "calculated output size too small (axis %d: %lld)", a,
                        (long long)p->out_size[a]);
    const int64_t lim = INT32_MAX;
    if (prod(p->in_size, p->dim) > lim || prod(p->out_size, p->dim) > lim ||
        p->batch * prod(p->in_size, p->dim) > (int64_t)1 << 40)
        return fail(TVDCN_ERR_UNSUPPORTED, "spatial extent exceeds 32-bit per-image indexing");
    if (p->batch > lim || p->in_channels > 1 << 20 || p->out_channels > 1 << 20)
        return fail(TVDCN_ERR_UNSUPPORTED, "batch / channel count too large");
    return TVDCN_OK;
}

GeoHost make_geo_host(const tvdcn_problem *p) {
    GeoHost g;
    memset(&g, 0, sizeof(g));
    g.dim = p->dim;
    g.B = (int)p->batch;
    g.Cs = (int)(p->transposed ? p->out_channels : p->in_channels);
    g.Cd = (int)(p->transposed ? p->in_channels : p->out_channels);
    g.groups = p->groups;
    g.og = p->offset_groups;
    g.mg = p->mask_groups;
    g.K = 1;
    g.S = 1;
    g.P = 1;
    for (int a = 0; a < p->dim; ++a) {
        g.img[a] = (int)(p->transposed ? p->out_size[a] : p->in_size[a]);
        g.grid[a] = (int)(p->transposed ? p->in_size[a] : p->out_size[a]);
        g.ker[a] = p->kernel[a];
        g.stride[a] = p->stride[a];
        g.pad[a] = p->padding[a];
        g.dil[a] = p->dilation[a];
        g.K *= g.ker[a];
        g.S *= g.img[a];
        g.P *= g.grid[a];
    }
    return g;
}

// One status word per device, living in the library's own device memory.
__device__ int g_tc_status;

int *device_status_word() {
    static int *cached[64] = {nullptr};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    if (cached[dev] == nullptr) {
        void *addr = nullptr;
        if (cudaGetSymbolAddress(&addr, g_tc_status) != cudaSuccess) return nullptr;
        cached[dev] = (int *)addr;
    }
    return cached[dev];
}

// Host words that mirror the status word, one per device (tvdcn_b200_watch_status); and whether this thread's latest
// call has a kernel that publishes an earlier call's code there.
static std::atomic<int *> g_host_word[64];
static thread_local bool t_published = false;

static cudaError_t current_status(Status *st) {
    int dev = 0;
    st->device = device_status_word();
    if (st->device == nullptr || cudaGetDevice(&dev) != cudaSuccess) return cudaErrorInvalidDevice;
    st->host = g_host_word[dev].load(std::memory_order_acquire);
    return cudaSuccess;
}

// One call on the tensor-core kernels: pointers into the workspace, and the preparations, which all go into one
// launch in front of the kernels.
struct TcCall {
    const tvdcn_problem *p;
    GeoHost g;              // padded geometry
    const Plan &pl;
    char *ws;
    Status status{};
    Stager stage;
    const float *offset = nullptr, *mask = nullptr, *bias = nullptr;

    TcCall(const tvdcn_problem *p_, const GeoHost &real, const Plan &pl_, char *ws_)
        : p(p_), g(tc_geometry(real)), pl(pl_), ws(ws_) {}
    void *at(size_t buf) const { return buf == NO_BUF ? nullptr : ws + buf; }
    void parts(const size_t (&buf)[3], void *(&out)[3]) const {
        for (int q = 0; q < 3; ++q) out[q] = at(buf[q]);
    }
    void stage_image(const void *img) {
        stage.image(img, at(pl.img_cl), g, p->dtype == TVDCN_F32 ? 4 : 2, static_cast<unsigned *>(at(pl.img_max)));
    }
    void stage_weight(const void *weight, bool kd) {
        void *w[3];
        parts(kd ? pl.w_pack_kd : pl.w_pack, w);
        stage.pack(weight, w, g, p->dtype, mode_mat_parts(pl.mode), kd);
        if (!kd && pl.sg_counters > 0) stage.zero(at(pl.sg_arrived), (int64_t)(pl.sg_counters * sizeof(unsigned)));
    }
    void stage_aux(const void *off, const void *msk, const void *bia) {
        const int64_t points = (int64_t)g.B * g.K * g.P;
        auto widen = [&](const void *src, size_t buf, int64_t n, unsigned *maxima = nullptr) -> const float * {
            if (src == nullptr || buf == NO_BUF) return static_cast<const float *>(src);
            stage.widen(src, at(buf), p->aux_dtype, n, maxima);
            return static_cast<const float *>(at(buf));
        };
        offset = widen(off, pl.off32, points * g.og * g.dim);
        unsigned *maxima = static_cast<unsigned *>(at(pl.mask_max));
        mask = widen(msk, pl.mask32, points * g.mg, maxima);
        if (msk != nullptr && msk == mask && maxima != nullptr) stage.max_abs(msk, maxima, points * g.mg);
        bias = widen(bia, pl.bias32, p->out_channels);
    }
    ColumnRange range() const {
        return {static_cast<unsigned *>(at(pl.img_max)), static_cast<unsigned *>(at(pl.mask_max)), pl.n_img_max, pl.n_mask_max};
    }
    cudaError_t prepare(cudaStream_t stream) {
        cudaError_t e = current_status(&status);
        if (e == cudaSuccess) e = stage.launch(status, stream);
        t_published = !stage.empty();
        return e;
    }
    cudaError_t sample_gemm(void *out, cudaStream_t stream) const {
        void *w[3];
        parts(pl.w_pack, w);
        return launch_sample_gemm_tc(g, pl.mode, at(pl.img_cl), w, offset, mask, bias, range(), out,
                                     static_cast<float *>(at(pl.sg_partial)), static_cast<unsigned *>(at(pl.sg_arrived)),
                                     status, stream);
    }
    // scatter_out (data type of the problem, [B, Cs, *img], may be null) receives the scattered image plus bias;
    // goff / gmask are zeroed f32 accumulators, may be null
    cudaError_t gemm_scatter(const void *dense, void *scatter_out, void *goff, void *gmask, cudaStream_t stream) const {
        void *w[3];
        parts(pl.w_pack_kd, w);
        float *acc = scatter_out != nullptr ? static_cast<float *>(at(pl.img_grad_cl)) : nullptr;
        const bool want_coord = goff != nullptr || gmask != nullptr;
        cudaError_t e = launch_gemm_scatter_tc(g, pl.mode, dense, w, want_coord ? at(pl.img_cl) : nullptr, offset, mask, acc,
                                               (float *)goff, (float *)gmask, status, stream);
        if (e == cudaSuccess && scatter_out != nullptr)
            e = launch_from_channels_last_bias(acc, bias, scatter_out, p->dtype, g, stream);
        return e;
    }
    cudaError_t channel_sum(const void *x, int C, int S, void *out, cudaStream_t stream) const {
        return launch_dense_pass(x, p->dtype, 0, nullptr, g.B, C, S, 0, (float *)at(pl.sum_partial),
                                 (unsigned *)at(pl.sum_done), out, p->aux_dtype, stream);
    }
    // Weight gradient into the staged accumulator and from there to grad_weight.  f32 data: the dense tensor is split
    // into bf16 parts first; the same pass takes its channel sums (bias gradient of the conv) where `sum_out` is given
    // and the pointer allows 16-byte loads, which *summed reports.
    cudaError_t sample_wgrad(const void *dense, void *grad_weight, void *sum_out, bool *summed, cudaStream_t stream) const {
        void *d[3] = {const_cast<void *>(dense), nullptr, nullptr};
        int pitch = g.P;
        cudaError_t e = cudaSuccess;
        *summed = false;
        if (pl.dense[0] != NO_BUF) {
            parts(pl.dense, d);
            pitch = pl.dense_pitch;
            if (p->dtype == TVDCN_F32) {
                *summed = sum_out != nullptr && reinterpret_cast<uintptr_t>(dense) % 16 == 0;
                e = launch_dense_pass(dense, p->dtype, mode_mat_parts(pl.mode_sw), d, g.B, g.Cd_r, g.P, pitch,
                                      (float *)at(pl.sum_partial), (unsigned *)at(pl.sum_done),
                                      *summed ? sum_out : nullptr, p->aux_dtype, stream);
            }
        }
        float *acc = static_cast<float *>(at(pl.gw_acc));
        if (e == cudaSuccess)
            e = launch_sample_wgrad_tc(g, pl.mode_sw, d, pitch, at(pl.img_cl), offset, mask, range(), acc, status, stream);
        if (e == cudaSuccess) e = launch_unpack_weight_grad(acc, grad_weight, p->dtype, g, stream);
        return e;
    }
};

// Waits on a barrier that nothing arrives on, with a small poll limit, and reports the time-out the way the
// tensor-core kernels do.
__global__ void bounded_wait_selftest_kernel(int *status, uint32_t max_polls) {
    __shared__ uint64_t bar;
    if (threadIdx.x == 0) {
        ptx::mbar_init(&bar, 1);
        ptx::fence_mbar_init();
    }
    __syncthreads();
    bool done = false;
    for (uint32_t i = 0; i < max_polls && !done; ++i) done = ptx::mbar_try_wait(&bar, 0);
    if (!done && threadIdx.x == 0) atomicExch(status, 900);
}

// What a call's first tensor-core kernel does in passing, for calls that launch none.
__global__ void publish_status_kernel(const Status status) { ptx::publish(status); }

}  // namespace tvdcn_b200

using namespace tvdcn_b200;

#define CUDA_TRY(expr)                                   \
    do {                                                 \
        cudaError_t e__ = (expr);                        \
        if (e__ != cudaSuccess) return cuda_fail(e__, #expr); \
    } while (0)

// The plan of a call.  Shapes that the tensor-core kernels take only with padding also run on the SIMT kernels, which
// need less workspace or none: a caller that brings no more than that gets those.
template <typename F>
static Plan plan_for(const tvdcn_problem *p, size_t workspace_bytes, F &&plan) {
    Plan pl = plan(p);
    if (pl.tensor && pl.wide && pl.total > workspace_bytes && p->engine == TVDCN_ENGINE_AUTO) {
        tvdcn_problem simt = *p;
        simt.engine = TVDCN_ENGINE_SIMT;
        pl = plan(&simt);
    }
    return pl;
}

extern "C" {

int tvdcn_b200_problem_finalize(tvdcn_problem *p) {
    int rc = check_problem(p);
    if (rc) return rc;
    for (int a = 0; a < 3; ++a) p->out_size[a] = 1;
    for (int a = 0; a < p->dim; ++a) {
        const int64_t in = p->in_size[a], k = p->kernel[a], s = p->stride[a], pd = p->padding[a],
                      d = p->dilation[a];
        if (!p->transposed) {
            const int64_t num = in + 2 * pd - (d * (k - 1) + 1);
            p->out_size[a] = num < 0 ? 0 : num / s + 1;
        } else {
            p->out_size[a] = (in - 1) * s - 2 * pd + d * (k - 1) + 1 + p->output_padding[a];
        }
    }
    for (int a = p->dim; a < 3; ++a) p->in_size[a] = 1;
    return check_sizes(p);
}

size_t tvdcn_b200_forward_workspace_bytes(const tvdcn_problem *p) {
    if (check_problem(p) || check_sizes(p)) return 0;
    return plan_forward(p).total;
}

size_t tvdcn_b200_backward_workspace_bytes(const tvdcn_problem *p) {
    if (check_problem(p) || check_sizes(p)) return 0;
    return plan_backward(p, true, true, true, true).total;
}

const char *tvdcn_b200_engine_name(const tvdcn_problem *p, int backward) {
    if (check_problem(p) || check_sizes(p)) return "invalid";
    const Plan pl = backward ? plan_backward(p, true, true, true, true) : plan_forward(p);
    return pl.tensor ? "tcgen05" : "simt";
}

static int check_ws(const Plan &pl, void *ws, size_t bytes) {
    if (pl.total == 0) return TVDCN_OK;
    if (ws == nullptr || bytes < pl.total)
        return fail(TVDCN_ERR_WORKSPACE, "workspace of %zu bytes required, %zu given", pl.total, bytes);
    if (reinterpret_cast<uintptr_t>(ws) % 256 != 0)
        return fail(TVDCN_ERR_WORKSPACE, "workspace must be 256-byte aligned");
    return TVDCN_OK;
}

static int check_forward_args(const tvdcn_problem *p, const void *input, const void *weight, const void *offset,
                              const void *mask, const void *output) {
    if (input == nullptr || weight == nullptr || output == nullptr)
        return fail(TVDCN_ERR_INVALID, "input, weight and output must not be NULL");
    if ((p->offset_groups > 0) != (offset != nullptr))
        return fail(TVDCN_ERR_INVALID, "offset pointer and offset_groups disagree");
    if ((p->mask_groups > 0) != (mask != nullptr))
        return fail(TVDCN_ERR_INVALID, "mask pointer and mask_groups disagree");
    return TVDCN_OK;
}

static int run_forward(const tvdcn_problem *p, const Plan &pl, const void *input, const void *weight, const void *offset,
                       const void *mask, const void *bias, void *output, void *workspace, cudaStream_t stream) {
    char *ws = (char *)workspace;
    const GeoHost g = make_geo_host(p);
    const int dt = p->dtype, aux = p->aux_dtype;
    t_published = false;

    if (pl.tensor) {
        TcCall tc(p, g, pl, ws);
        if (pl.tc_sg) tc.stage_image(input);
        tc.stage_weight(weight, pl.tc_gs);
        tc.stage_aux(offset, mask, bias);
        if (pl.tc_gs) tc.stage.zero(ws + pl.img_grad_cl, (int64_t)g.B * g.S * tc.g.Cs * (int64_t)sizeof(float));
        CUDA_TRY(tc.prepare(stream));
        if (pl.tc_sg)
            CUDA_TRY(tc.sample_gemm(output, stream));
        else
            CUDA_TRY(tc.gemm_scatter(input, output, nullptr, nullptr, stream));
        return TVDCN_OK;
    }

    if (!p->transposed) {
        CUDA_TRY(launch_sample_gemm(g, dt, aux, input, weight, offset, mask, bias, output, stream));
        return TVDCN_OK;
    }
    // transposed: output (= sampled image) starts as the bias and receives the scatter
    const int64_t n_out = (int64_t)g.B * g.Cs * g.S;
    void *acc = pl.img_acc != NO_BUF ? (void *)(ws + pl.img_acc) : output;
    CUDA_TRY(launch_fill_bias(dt, aux, bias, g.B, g.Cs, g.S, acc, stream));
    CUDA_TRY(launch_gemm_scatter(g, dt, aux, input, weight, offset, mask, nullptr, acc, nullptr, nullptr, stream));
    if (pl.img_acc != NO_BUF) CUDA_TRY(launch_cast_from_acc(dt, acc, output, n_out, stream));
    return TVDCN_OK;
}

int tvdcn_b200_deform_conv_forward(const tvdcn_problem *p, const void *input, const void *weight,
                                   const void *offset, const void *mask, const void *bias, void *output,
                                   void *workspace, size_t workspace_bytes, void *cuda_stream) {
    int rc = check_problem(p);
    if (rc) return rc;
    rc = check_sizes(p);
    if (rc) return rc;
    if (p->batch == 0) return TVDCN_OK;  // nothing to compute; empty tensors may have NULL storage
    rc = check_forward_args(p, input, weight, offset, mask, output);
    if (rc) return rc;
    const Plan pl = plan_for(p, workspace_bytes, [](const tvdcn_problem *q) { return plan_forward(q); });
    if (p->engine == TVDCN_ENGINE_TENSOR && !pl.tensor)
        return fail(TVDCN_ERR_UNSUPPORTED, "shape not covered by the tensor-core kernels: %s", pl.why_not);
    rc = check_ws(pl, workspace, workspace_bytes);
    if (rc) return rc;
    return run_forward(p, pl, input, weight, offset, mask, bias, output, workspace, (cudaStream_t)cuda_stream);
}

// Side stream of the backward pass: the scatter kernel does not depend on the weight-gradient kernel and the bias sum,
// so it is queued beside them and its CTAs fill the SMs that their last, partial wave leaves idle.  The weight gradient
// keeps the caller's stream and goes first: it is final early in the call, so its all-reduce can run under the rest of
// the scatter (the other way round its CTAs had to wait for whole waves of scatter CTAs to retire).  One stream and two events per host thread and device, created on first use and kept; fork and join are
// event waits, so the caller's stream still orders the whole call (and a capture of it picks both streams up).
// TVDCN_B200_OVERLAP=0 keeps everything on the caller's stream, and so does tvdcn_b200_timing_enable(1).
struct SideStream {
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    bool tried = false;
};
static SideStream *side_stream() {
    static thread_local SideStream per_device[64];
    static const bool enabled = [] {
        const char *v = getenv("TVDCN_B200_OVERLAP");
        return v == nullptr || v[0] != '0';
    }();
    // per-kernel timing wants every kernel alone on the GPU
    if (!enabled || g_timing.load(std::memory_order_relaxed)) return nullptr;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
    SideStream &s = per_device[dev];
    if (!s.tried) {
        s.tried = true;
        if (cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking) != cudaSuccess ||
            cudaEventCreateWithFlags(&s.fork, cudaEventDisableTiming) != cudaSuccess ||
            cudaEventCreateWithFlags(&s.join, cudaEventDisableTiming) != cudaSuccess) {
            s.stream = nullptr;
            (void)cudaGetLastError();
        }
    }
    return s.stream != nullptr ? &s : nullptr;
}

int tvdcn_b200_deform_conv_backward(const tvdcn_problem *p, const void *grad_output, const void *input,
                                    const void *weight, const void *offset, const void *mask, void *grad_input,
                                    void *grad_weight, void *grad_offset, void *grad_mask, void *grad_bias,
                                    void *workspace, size_t workspace_bytes, void *cuda_stream) {
    return tvdcn_b200_deform_conv_backward_ex(p, grad_output, input, weight, offset, mask, grad_input, grad_weight,
                                              grad_offset, grad_mask, grad_bias, workspace, workspace_bytes,
                                              cuda_stream, nullptr);
}

int tvdcn_b200_deform_conv_backward_ex(const tvdcn_problem *p, const void *grad_output, const void *input,
                                       const void *weight, const void *offset, const void *mask, void *grad_input,
                                       void *grad_weight, void *grad_offset, void *grad_mask, void *grad_bias,
                                       void *workspace, size_t workspace_bytes, void *cuda_stream,
                                       void *weight_grad_ready) {
    int rc = check_problem(p);
    if (rc) return rc;
    rc = check_sizes(p);
    if (rc) return rc;
    cudaStream_t stream = (cudaStream_t)cuda_stream;
    const GeoHost g = make_geo_host(p);
    const int dt = p->dtype, aux = p->aux_dtype;
    const size_t es = dtype_size(dt), as = dtype_size(aux);
    const int64_t n_w = (int64_t)g.Cd * (g.Cs / g.groups) * g.K;
    const int64_t n_off = (int64_t)g.B * g.og * g.K * g.dim * g.P;
    const int64_t n_mask = (int64_t)g.B * g.mg * g.K * g.P;
    const int64_t n_img = (int64_t)g.B * g.Cs * g.S;
    if (p->batch == 0) {
        if (grad_weight) CUDA_TRY(cudaMemsetAsync(grad_weight, 0, n_w * es, stream));
        if (grad_bias) CUDA_TRY(cudaMemsetAsync(grad_bias, 0, (size_t)p->out_channels * as, stream));
        if (weight_grad_ready) CUDA_TRY(cudaEventRecord((cudaEvent_t)weight_grad_ready, stream));
        return TVDCN_OK;  // empty batch: the sums over the batch are zero, empty tensors may be NULL
    }
    if (grad_output == nullptr || input == nullptr || weight == nullptr)
        return fail(TVDCN_ERR_INVALID, "grad_output, input and weight must not be NULL");
    if ((p->offset_groups > 0) != (offset != nullptr))
        return fail(TVDCN_ERR_INVALID, "offset pointer and offset_groups disagree");
    if ((p->mask_groups > 0) != (mask != nullptr))
        return fail(TVDCN_ERR_INVALID, "mask pointer and mask_groups disagree");
    if (grad_offset != nullptr && offset == nullptr)
        return fail(TVDCN_ERR_INVALID, "grad_offset requested without offset");
    if (grad_mask != nullptr && mask == nullptr) return fail(TVDCN_ERR_INVALID, "grad_mask requested without mask");
    const Plan pl = plan_for(p, workspace_bytes, [&](const tvdcn_problem *q) {
        return plan_backward(q, grad_input != nullptr, grad_weight != nullptr, grad_offset != nullptr, grad_mask != nullptr);
    });
    if (p->engine == TVDCN_ENGINE_TENSOR && !pl.tensor)
        return fail(TVDCN_ERR_UNSUPPORTED, "shape not covered by the tensor-core kernels: %s", pl.why_not);
    rc = check_ws(pl, workspace, workspace_bytes);
    if (rc) return rc;
    char *ws = (char *)workspace;
    t_published = false;
    const size_t acs = dtype_size(acc_dtype(dt));
    // accumulation targets: the outputs themselves when they already have the accumulation type
    void *gw_acc = grad_weight ? (pl.gw_acc != NO_BUF ? (void *)(ws + pl.gw_acc) : grad_weight) : nullptr;
    void *goff_acc = grad_offset ? (pl.goff_acc != NO_BUF ? (void *)(ws + pl.goff_acc) : grad_offset) : nullptr;
    void *gmask_acc = grad_mask ? (pl.gmask_acc != NO_BUF ? (void *)(ws + pl.gmask_acc) : grad_mask) : nullptr;
    // sampled image and dense tensor: conv: input and grad_output, transposed: grad_output and input
    const void *img = p->transposed ? grad_output : input, *dense = p->transposed ? input : grad_output;
    void *gi_acc = nullptr;   // conv on the SIMT kernels: where grad_input is accumulated
    if (!p->transposed && grad_input && !pl.tc_gs) gi_acc = pl.img_acc != NO_BUF ? (void *)(ws + pl.img_acc) : grad_input;

    // The weight-gradient kernel reads 16-bit dense tensors by TMA straight from the caller's pointer, which must
    // then sit on a 16-byte boundary (a tensor view with a storage offset may not): the SIMT kernel takes over.
    const bool tc_sw = pl.tc_sw && (pl.dense[0] != NO_BUF || (reinterpret_cast<uintptr_t>(dense) & 15) == 0);

    TcCall tc(p, g, pl, ws);
    if (pl.tensor) {
        // The caller may vouch that the forward call's staging of `input` is still at the start of this workspace
        // (only where the forward call for this problem stages the image at all, and at the same offset: with a workspace
        // too small for its plan, which may still do for this call's, it ran on the SIMT kernels and staged nothing; and f16 rows that
        // TMA cannot read make the weight gradient alone wide, whose maxima the forward call had no use for).
        bool staged = false;
        if ((p->flags & TVDCN_FLAG_REUSE_STAGED_INPUT) && !p->transposed) {
            const Plan fwd = plan_for(p, workspace_bytes, [](const tvdcn_problem *q) { return plan_forward(q); });
            staged = fwd.img_cl != NO_BUF && fwd.img_cl == pl.img_cl && fwd.total <= workspace_bytes &&
                     (pl.img_max == NO_BUF || pl.img_max == fwd.img_max);
        }
        if (!staged && (pl.tc_sg || tc_sw || goff_acc || gmask_acc)) tc.stage_image(img);
        if (pl.tc_gs) tc.stage_weight(weight, true);
        if (pl.tc_sg) tc.stage_weight(weight, false);
        tc.stage_aux(offset, mask, nullptr);
        if (tc_sw && p->dtype != TVDCN_F32 && pl.dense[0] != NO_BUF)
            tc.stage.pitch(dense, ws + pl.dense[0], (int64_t)g.B * g.Cd, g.P, pl.dense_pitch);
        if (grad_bias) tc.stage.zero(ws + pl.sum_done, (int64_t)p->out_channels * (int64_t)sizeof(unsigned));
    }
    auto zero = [&](void *ptr, int64_t bytes) { if (ptr != nullptr) tc.stage.zero(ptr, bytes); };
    zero(gw_acc, pl.tc_sw ? (int64_t)g.Cd * (tc.g.Cs / g.groups) * g.K * 4 : n_w * (int64_t)acs);
    zero(goff_acc, n_off * (int64_t)acs);
    zero(gmask_acc, n_mask * (int64_t)acs);
    zero(gi_acc, n_img * (int64_t)acs);
    // Fork: the scatter kernel on the side stream when both sides run on the tensor cores.
    SideStream *side = (tc_sw && gw_acc && (pl.tc_gs || pl.tc_sg)) ? side_stream() : nullptr;
    cudaStream_t sstream = side != nullptr ? side->stream : stream;
    // A large scatter accumulator is zeroed under the weight gradient; below 32 MB (5 us) the launch costs more.
    const int64_t acc_bytes = pl.img_grad_cl != NO_BUF ? (int64_t)g.B * g.S * tc.g.Cs * 4 : 0;
    const bool zero_later = side != nullptr && acc_bytes > (32 << 20);
    if (acc_bytes > 0 && !zero_later) tc.stage.zero(ws + pl.img_grad_cl, acc_bytes);
    CUDA_TRY(tc.prepare(stream));
    if (side != nullptr) {
        CUDA_TRY(cudaEventRecord(side->fork, stream));
        CUDA_TRY(cudaStreamWaitEvent(sstream, side->fork, 0));
    }
    auto weight_and_bias = [&]() -> int {
        bool summed = false;
        if (gw_acc && tc_sw)
            CUDA_TRY(tc.sample_wgrad(dense, grad_weight, p->transposed ? nullptr : grad_bias, &summed, stream));
        else if (gw_acc)
            CUDA_TRY(launch_sample_wgrad(g, dt, aux, dense, img, offset, mask, gw_acc, stream));
        if (grad_bias && !summed) {
            const int c = (int)p->out_channels, n = p->transposed ? g.S : g.P;
            if (pl.tensor)
                CUDA_TRY(tc.channel_sum(grad_output, c, n, grad_bias, stream));
            else
                CUDA_TRY(launch_channel_sum(dt, aux, grad_output, g.B, c, n, grad_bias, stream));
        }
        if (gw_acc && pl.gw_acc != NO_BUF && !tc_sw)
            CUDA_TRY(launch_cast_from_acc(dt, gw_acc, grad_weight, n_w, stream));
        if (weight_grad_ready) CUDA_TRY(cudaEventRecord((cudaEvent_t)weight_grad_ready, stream));
        return TVDCN_OK;
    };
    if ((rc = weight_and_bias()) != TVDCN_OK) return rc;
    // scatter and coordinate gradients; the transposed conv's grad_input is a sample -> GEMM
    if (zero_later) {
        Stager later;
        later.zero(ws + pl.img_grad_cl, acc_bytes);
        CUDA_TRY(later.launch(tc.status, sstream));
    }
    if (pl.tc_gs)
        CUDA_TRY(tc.gemm_scatter(dense, p->transposed ? nullptr : grad_input, goff_acc, gmask_acc, sstream));
    else if (gi_acc || goff_acc || gmask_acc)
        CUDA_TRY(launch_gemm_scatter(g, dt, aux, dense, weight, offset, mask, img, gi_acc, goff_acc, gmask_acc, sstream));
    if (p->transposed && grad_input) {
        if (pl.tc_sg)
            CUDA_TRY(tc.sample_gemm(grad_input, sstream));
        else
            CUDA_TRY(launch_sample_gemm(g, dt, aux, img, weight, offset, mask, nullptr, grad_input, sstream));
    }
    if (side != nullptr) {  // join
        CUDA_TRY(cudaEventRecord(side->join, sstream));
        CUDA_TRY(cudaStreamWaitEvent(stream, side->join, 0));
    }
    if (gi_acc && pl.img_acc != NO_BUF) CUDA_TRY(launch_cast_from_acc(dt, gi_acc, grad_input, n_img, stream));
    if (goff_acc && pl.goff_acc != NO_BUF) CUDA_TRY(launch_cast_from_acc(aux, goff_acc, grad_offset, n_off, stream));
    if (gmask_acc && pl.gmask_acc != NO_BUF)
        CUDA_TRY(launch_cast_from_acc(aux, gmask_acc, grad_mask, n_mask, stream));
    return TVDCN_OK;
}

int tvdcn_b200_mask_softmax_forward(int32_t dtype, int64_t batch, int64_t mask_groups, int64_t taps,
                                    int64_t spatial, const void *in, void *out, void *cuda_stream) {
    if (dtype < TVDCN_F32 || dtype > TVDCN_BF16) return fail(TVDCN_ERR_INVALID, "unknown dtype %d", dtype);
    if (batch < 0 || mask_groups <= 0 || taps <= 0 || spatial < 0 || taps > INT32_MAX)
        return fail(TVDCN_ERR_INVALID, "mask_softmax: bad extents");
    if (batch * spatial == 0) return TVDCN_OK;
    if (in == nullptr || out == nullptr) return fail(TVDCN_ERR_INVALID, "mask_softmax: NULL pointer");
    CUDA_TRY(launch_mask_softmax_fwd(dtype, batch * mask_groups, (int)taps, spatial, in, out,
                                     (cudaStream_t)cuda_stream));
    return TVDCN_OK;
}

int tvdcn_b200_mask_softmax_backward(int32_t dtype, int64_t batch, int64_t mask_groups, int64_t taps,
                                     int64_t spatial, const void *grad_out, const void *out, void *grad_in,
                                     void *cuda_stream) {
    if (dtype < TVDCN_F32 || dtype > TVDCN_BF16) return fail(TVDCN_ERR_INVALID, "unknown dtype %d", dtype);
    if (batch < 0 || mask_groups <= 0 || taps <= 0 || spatial < 0 || taps > INT32_MAX)
        return fail(TVDCN_ERR_INVALID, "mask_softmax: bad extents");
    if (batch * spatial == 0) return TVDCN_OK;
    if (grad_out == nullptr || out == nullptr || grad_in == nullptr)
        return fail(TVDCN_ERR_INVALID, "mask_softmax: NULL pointer");
    CUDA_TRY(launch_mask_softmax_bwd(dtype, batch * mask_groups, (int)taps, spatial, grad_out, out, grad_in,
                                     (cudaStream_t)cuda_stream));
    return TVDCN_OK;
}

int tvdcn_b200_selftest_bounded_wait(int max_polls, void *cuda_stream) {
    if (max_polls < 1 || max_polls > 4096) return fail(TVDCN_ERR_INVALID, "max_polls must be in [1, 4096]");
    int *status = device_status_word();
    if (status == nullptr) return fail(TVDCN_ERR_CUDA, "status word not found");
    count_launch();
    bounded_wait_selftest_kernel<<<1, 32, 0, (cudaStream_t)cuda_stream>>>(status, (uint32_t)max_polls);
    CUDA_TRY(cudaGetLastError());
    return TVDCN_OK;
}

int tvdcn_b200_cuda_version(void) { return CUDART_VERSION; }

const char *tvdcn_b200_cuda_arch_flags(void) { return "sm_100a"; }

const char *tvdcn_b200_last_error(void) { return g_err; }

void tvdcn_b200_timing_enable(int on) { g_timing.store(on ? 1 : 0, std::memory_order_relaxed); }

size_t tvdcn_b200_timing_report(char *buf, size_t cap) {
    std::vector<TimedLaunch> taken;
    {
        std::lock_guard<std::mutex> lk(g_timing_mu);
        taken.swap(g_timed);
    }
    struct Agg { uint64_t n = 0; double ms = 0; };
    std::map<std::string, Agg> agg;
    for (auto &t : taken) {
        float ms = 0.f;
        if (cudaEventSynchronize(t.stop) == cudaSuccess && cudaEventElapsedTime(&ms, t.start, t.stop) == cudaSuccess) {
            Agg &a = agg[t.name];
            a.n += 1;
            a.ms += ms;
        }
        cudaEventDestroy(t.start);
        cudaEventDestroy(t.stop);
    }
    std::string out;
    for (auto &kv : agg) {
        char line[160];
        snprintf(line, sizeof(line), "%s %llu %.6f\n", kv.first.c_str(), (unsigned long long)kv.second.n, kv.second.ms);
        out += line;
    }
    if (buf != nullptr && cap > 0) {
        const size_t n = out.size() < cap - 1 ? out.size() : cap - 1;
        memcpy(buf, out.data(), n);
        buf[n] = 0;
    }
    return out.size();
}

int tvdcn_b200_device_status(void) {
    int *word = device_status_word();
    if (word == nullptr) return -1;
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    int value = 0;
    if (cudaMemcpy(&value, word, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return -1;
    if (value != 0) cudaMemset(word, 0, sizeof(int));
    return value;
}

const int *tvdcn_b200_device_status_address(void) { return device_status_word(); }

int tvdcn_b200_publish_status(int *host_word_device_ptr, void *cuda_stream) {
    if (host_word_device_ptr == nullptr) return fail(TVDCN_ERR_INVALID, "host_word_device_ptr is NULL");
    Status status;
    CUDA_TRY(current_status(&status));
    const bool published = t_published;
    t_published = false;
    if (published && status.host == host_word_device_ptr) return TVDCN_OK;   // the call's own kernels did it
    status.host = host_word_device_ptr;
    publish_status_kernel<<<1, 1, 0, (cudaStream_t)cuda_stream>>>(status);
    CUDA_TRY(cudaGetLastError());
    return TVDCN_OK;
}

int tvdcn_b200_watch_status(int *host_word_device_ptr) {
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(TVDCN_ERR_UNSUPPORTED, "device index %d", dev);
    g_host_word[dev].store(host_word_device_ptr, std::memory_order_release);
    return TVDCN_OK;
}

uint64_t tvdcn_b200_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

}  // extern "C"

// ---- forward without a caller-provided workspace ---------------------------------------------------------
// Scratch for tvdcn_b200_deform_conv_forward_static.  The array lives in this library's device image: every
// GPU that loads the library keeps these bytes until the process exits.  In host code the name below is only
// a handle for cudaGetSymbolAddress -- it is not a device address and must never be handed to a kernel.
#define TVDCN_STATIC_SCRATCH_BYTES (16u << 20)
static __device__ __align__(256) unsigned char g_static_scratch[TVDCN_STATIC_SCRATCH_BYTES];

// Device address of the scratch array on the current device; looked up once per device.
static cudaError_t static_scratch_address(void **out) {
    static void *cached[64] = {nullptr};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (cached[dev] == nullptr) {
        void *addr = nullptr;
        e = cudaGetSymbolAddress(&addr, g_static_scratch);
        if (e != cudaSuccess) return e;
        cached[dev] = addr;
    }
    *out = cached[dev];
    return cudaSuccess;
}

extern "C" {

size_t tvdcn_b200_static_scratch_bytes(void) { return TVDCN_STATIC_SCRATCH_BYTES; }

int tvdcn_b200_deform_conv_forward_static(const tvdcn_problem *p, const void *input, const void *weight,
                                          const void *offset, const void *mask, const void *bias, void *output,
                                          void *cuda_stream) {
    int rc = check_problem(p);
    if (rc) return rc;
    rc = check_sizes(p);
    if (rc) return rc;
    if (p->batch == 0) return TVDCN_OK;
    rc = check_forward_args(p, input, weight, offset, mask, output);
    if (rc) return rc;
    // The plan is made for the scratch there is: without shared tiles where their partial sums do not fit, and on the
    // SIMT kernels where a padded shape does not fit at all.
    Plan pl = plan_forward(p);
    if (pl.total > TVDCN_STATIC_SCRATCH_BYTES)
        pl = plan_for(p, TVDCN_STATIC_SCRATCH_BYTES, [](const tvdcn_problem *q) { return plan_forward(q, false); });
    if (p->engine == TVDCN_ENGINE_TENSOR && !pl.tensor)
        return fail(TVDCN_ERR_UNSUPPORTED, "shape not covered by the tensor-core kernels: %s", pl.why_not);
    if (pl.total > TVDCN_STATIC_SCRATCH_BYTES)
        return fail(TVDCN_ERR_WORKSPACE,
                    "this problem needs %zu bytes of scratch, more than the %u bytes built into the library; use "
                    "tvdcn_b200_deform_conv_forward with a workspace of your own",
                    pl.total, (unsigned)TVDCN_STATIC_SCRATCH_BYTES);
    void *scratch = nullptr;
    if (pl.total > 0) {
        const cudaError_t e = static_scratch_address(&scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(static scratch)");
    }
    // The forward kernels overwrite every scratch byte they later read (staged image, packed weights) and
    // zero the scatter accumulator themselves, so nothing left by an earlier call can leak into this one.
    return run_forward(p, pl, input, weight, offset, mask, bias, output, scratch, (cudaStream_t)cuda_stream);
}

}  // extern "C"
