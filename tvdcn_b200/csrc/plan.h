// Engine choice and workspace layout of one forward / backward call (internal).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "../../include/tvdcn_b200.h"
#include "kernels.h"

namespace tvdcn_b200 {

constexpr size_t NO_BUF = (size_t)-1;

struct Plan {
    bool tensor = false;           // at least one primitive runs on the tensor-core (tcgen05) kernels
    bool tc_sg = false;            // sample -> GEMM on tensor cores
    bool tc_gs = false;            // GEMM -> scatter / coordinate gradients on tensor cores
    bool tc_sw = false;            // sampled weight gradient on tensor cores
    bool wide = false;             // a shape or type that needs padding or widening (see the modes)
    int mode = 0, mode_sw = 0;     // TC_* mode of tc_sg and tc_gs, and of tc_sw
    const char *why_not = "";      // reason the tensor-core kernels were not chosen
    size_t total = 0;              // workspace bytes
    // accumulation buffers for 16-bit outputs (byte offsets into the workspace)
    size_t img_acc = NO_BUF;       // SIMT path: sampled-image-shaped accumulator (grad_input / transposed output)
    size_t gw_acc = NO_BUF;        // f32 weight gradient: [Cd, csg, K] for the SIMT kernel, [g][tap][d'][s'] for the tensor-core one
    size_t goff_acc = NO_BUF;
    size_t gmask_acc = NO_BUF;
    // tensor path: staged copies; weights and dense tensor in as many 16-bit parts as the mode has
    size_t img_cl = NO_BUF;        // sampled image, channels-last, data type of the problem
    size_t w_pack[3] = {NO_BUF, NO_BUF, NO_BUF};      // weights packed [g][tap][d'][s']
    size_t w_pack_kd[3] = {NO_BUF, NO_BUF, NO_BUF};   // weights packed [g][tap][s'][d']
    size_t dense[3] = {NO_BUF, NO_BUF, NO_BUF};       // dense tensor, rows dense_pitch apart (absent: the caller's own)
    int dense_pitch = 0;
    size_t img_grad_cl = NO_BUF;   // f32 channels-last accumulator of the scatter
    size_t img_max = NO_BUF, mask_max = NO_BUF;   // see ColumnRange: maxima of the image's and the mask's blocks
    int n_img_max = 0, n_mask_max = 0;
    size_t off32 = NO_BUF, mask32 = NO_BUF, bias32 = NO_BUF;   // 16-bit offset / mask / bias widened to f32
    size_t sg_partial = NO_BUF, sg_arrived = NO_BUF, sg_counters = 0;   // sample -> GEMM: tiles shared between CTAs
    size_t sum_partial = NO_BUF, sum_done = NO_BUF;   // partial sums of the bias gradient and their arrival counters
};

inline size_t align_up(size_t v, size_t a = 256) { return (v + a - 1) / a * a; }

// share_tiles: sample -> GEMM tiles may be shared between CTAs, whose partial sums then take up to 39 MB of workspace
Plan plan_forward(const tvdcn_problem *p, bool share_tiles = true);
Plan plan_backward(const tvdcn_problem *p, bool want_input, bool want_weight, bool want_offset, bool want_mask);

GeoHost make_geo_host(const tvdcn_problem *p);
int fail(int code, const char *fmt, ...);
int cuda_fail(cudaError_t e, const char *what);

// The geometry the tensor-core kernels work on: channels padded as GeoHost describes.
GeoHost tc_geometry(const GeoHost &g);

// ---- staging (sm100_staging.cu) ------------------------------------------------------------------------
enum : int { STAGE_IMAGE, STAGE_PACK, STAGE_ZERO, STAGE_WIDEN, STAGE_PITCH, STAGE_MAX };
struct StageJob {
    const void *src;
    // part: STAGE_PACK: one tensor per part; STAGE_IMAGE (f16), STAGE_WIDEN (may be null), STAGE_MAX: [0] = the blocks' maxima
    void *dst, *part[3];
    int64_t n;
    int kind, end_block;           // the job's blocks end before this one
    int dtype, elem_bytes, wide, kd;
    int C, c_pad, gran, gran_pad, S, K, cdg, cdg_pad;
};
struct StageList {
    static constexpr int MAX = 14;
    int n;
    Status status;
    StageJob job[MAX];
};
// Collects the preparations of one call and runs them as one launch.
class Stager {
   public:
    // + the row of zeros behind it; maxima (f16, may be null): image_blocks values
    void image(const void *src, void *dst, const GeoHost &h, int elem_bytes, unsigned *maxima);
    static int64_t image_blocks(const GeoHost &h) { return (int64_t)h.B * ((h.S + 63) / 64) * (h.Cs / 64); }
    void pack(const void *weight, void *const *parts, const GeoHost &h, int dtype, int n_parts, bool kd);
    void zero(void *dst, int64_t bytes);                                        // bytes: a multiple of 4
    void widen(const void *src, void *dst, int dtype, int64_t n, unsigned *maxima = nullptr);   // 16-bit -> f32
    static int64_t widen_blocks(int64_t n);
    void pitch(const void *src, void *dst, int64_t rows, int P, int pitch);     // 16-bit rows, `pitch` apart
    void max_abs(const void *src, unsigned *maxima, int64_t n);                 // f32, widen_blocks values
    cudaError_t launch(const Status &status, cudaStream_t stream);
    bool empty() const { return list_.n == 0; }

   private:
    StageJob *add(int kind, int64_t blocks);
    StageList list_{};
    int64_t blocks_ = 0;
    cudaError_t error_ = cudaSuccess;
};
cudaError_t launch_from_channels_last_bias(const float *src, const float *bias, void *dst, int dst_dtype, const GeoHost &h,
                                           cudaStream_t stream);
// staged weight gradient of the tensor-core kernel, [g][tap][d'][s'] f32 -> [Cd, csg, K] in the data type `dtype`
cudaError_t launch_unpack_weight_grad(const float *staged, void *gw, int dtype, const GeoHost &h, cudaStream_t stream);
// One read of a [B, C, P] tensor (f32, f16 or bf16): its bf16 parts (f32 data; n_parts 0: none) and / or the sum over
// batch and space per channel (sum_out, may be null).  partial: dense_sum_scratch_floats values; done: C zeroed counters.
int64_t dense_sum_scratch_floats(int B, int C, int P);
cudaError_t launch_dense_pass(const void *src, int dtype, int n_parts, void *const *parts, int B, int C, int P, int pitch,
                              float *partial, unsigned *done, void *sum_out, int sum_dtype, cudaStream_t stream);

// ---- tensor-core kernels (sm100_*.cu); all take the padded geometry ---------------------------------------
// A configuration is returned for every problem that the launcher below it takes, and for no other.
bool fwd_tc_config(const GeoHost &h, int mode, int *bn, int *stages);
cudaError_t launch_sample_gemm_tc(const GeoHost &h, int mode, const void *img_cl, void *const *w_parts,
                                  const float *offset, const float *mask, const float *bias, const ColumnRange &range,
                                  void *out, float *partial, unsigned *arrived, const Status &status, cudaStream_t stream);
void fwd_tc_workspace(const GeoHost &h, int mode, int bn, size_t *partial_bytes, size_t *counters);   // partial sums of shared tiles
bool wgrad_tc_config(const GeoHost &h, int mode, int *n_sub, int *m_tiles, int *stages);
cudaError_t launch_sample_wgrad_tc(const GeoHost &h, int mode, void *const *dense_parts, int pitch, const void *img_cl,
                                   const float *offset, const float *mask, const ColumnRange &range, float *gw,
                                   const Status &status, cudaStream_t stream);
bool dgrad_tc_config(const GeoHost &h, int mode, int *tb, int *nacc, int *b_stages);
cudaError_t launch_gemm_scatter_tc(const GeoHost &h, int mode, const void *dense, void *const *w_parts,
                                   const void *img_cl, const float *offset, const float *mask, float *img_grad_cl,
                                   float *goff, float *gmask, const Status &status, cudaStream_t stream);

// Address of the per-device status word the tensor-core kernels report failed bounded waits in.
int *device_status_word();

}  // namespace tvdcn_b200
