// Host-side launchers of the device kernels (internal; the public surface is include/tvdcn_b200.h).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace tvdcn_b200 {

// Runtime-dimension geometry; converted to Geo<DIM> at launch.
struct GeoHost {
    int dim;
    int B, Cs, Cd, groups, og, mg, K, S, P;
    int img[3], grid[3], ker[3], stride[3], pad[3], dil[3];
    // Only the tensor-core kernels look at these: their chunks of 64 channels must not straddle a convolution,
    // offset or mask group, so tc_geometry() pads every run of `gran` sampled channels that share their groups to
    // gran_pad (in the staged image and weights) and the dense channels of a group to a multiple of 64.  Cs and Cd
    // then count padded channels, Cs_r and Cd_r those of the caller's tensors.
    int Cs_r, Cd_r, gran, gran_pad;
};

enum : int { DT_F32 = 0, DT_F64 = 1, DT_F16 = 2, DT_BF16 = 3 };

inline size_t dtype_size(int dt) { return dt == DT_F64 ? 8 : (dt == DT_F32 ? 4 : 2); }
// accumulation type that goes with a data type: double for f64, float otherwise
inline int acc_dtype(int dt) { return dt == DT_F64 ? DT_F64 : DT_F32; }

// How the 16-bit tensor-core operands are derived from the user's data type.  A sampled column or a matrix operand
// (weights, dense tensor) travels as one or more 16-bit parts of decreasing magnitude whose sum is the value:
//   TC_BF16, TC_F16   16-bit data; columns blended and rounded in that type: one part, one MMA per K step
//   TC_SPLIT          f32 data as bf16 hi + lo (about 16 bits): three MMAs (hi*hi, lo*hi, hi*lo)
//   TC_*_WIDE         the precision of the SIMT kernels, for the shapes and types that only those used to take:
//                     16-bit data with columns blended in f32 and kept in two parts (the matrix operand is exact in
//                     one): two MMAs; f32 data in three bf16 parts (all 24 bits): the six products above 2^-24.
//                     f16 parts have f16's range: see ColumnRange
// For f32 data the products of the leading parts have accumulators of their own: the tensor core's f32 accumulation
// rounds toward zero, by half an ulp of the accumulator per MMA on average, so the small products must not touch the
// large sum (16-bit results do not see it).
enum : int { TC_BF16 = 0, TC_F16 = 1, TC_SPLIT = 2, TC_BF16_WIDE = 3, TC_F16_WIDE = 4, TC_F32_WIDE = 5 };
inline int mode_col_parts(int mode) { return mode == TC_F32_WIDE ? 3 : (mode >= TC_SPLIT ? 2 : 1); }
inline int mode_mat_parts(int mode) { return mode == TC_F32_WIDE ? 3 : (mode == TC_SPLIT ? 2 : 1); }
inline bool mode_f32(int mode) { return mode == TC_SPLIT || mode == TC_F32_WIDE; }

// What bounds the columns of TC_F16_WIDE: the largest finite |image value| and |mask|, as float bits, one value per block
// of the staging kernel that took them.  A column is at most their product, which may pass f16's 65504, or lie so low that
// the second part falls below f16's 2^-24.  The kernels multiply the mask by the power of two that brings the product
// just below 2^15, and their sums by its inverse: no column overflows, and a column keeps 22 bits down to 2^-18 of the
// largest possible one, below that an absolute error of 2^-40 of it.
// It costs 2 us of the 50 that one 256-channel 67 x 101 image takes (maxima 0.6, their reduction 1.0, the factor 0.4).
struct ColumnRange {
    const unsigned *img, *mask;
    int n_img, n_mask;             // n_mask 0: no mask (factor 1)
};

// Where a kernel whose bounded wait ran out leaves a code: the device word, and the host word (mapped pinned memory,
// may be null) that the PyTorch front end looks at.
struct Status {
    int *device;
    int *host;
};

void count_launch(int n = 1);

// Put one of these on the stack around a kernel launch: it counts the launch and, while kernel timing is
// switched on (tvdcn_b200_timing_enable), brackets it with CUDA events on the launching stream.
struct LaunchScope {
    LaunchScope(const char *name, cudaStream_t stream);
    ~LaunchScope();
    LaunchScope(const LaunchScope &) = delete;
    LaunchScope &operator=(const LaunchScope &) = delete;

   private:
    const char *name_;
    cudaStream_t stream_;
    cudaEvent_t start_ = nullptr;
};

// ---- generic SIMT kernels (generic.cu) -------------------------------------------------
// dense[b, d, p] = bias[d] + sum_{s', tap} W[d, s', tap] * mask * sample(img[b, s], pos)
cudaError_t launch_sample_gemm(const GeoHost &g, int dtype, int aux_dtype, const void *img, const void *weight,
                               const void *offset, const void *mask, const void *bias, void *dense_out,
                               cudaStream_t stream);

// col = W^T * dense per group, consumed in registers:
//   img_grad_acc[b, s, corners] += col * mask * corner weight          (if img_grad_acc)
//   goff_acc[b, og, tap, axis, p] += col * mask * d sample / d axis     (if goff_acc; needs img)
//   gmask_acc[b, mg, tap, p]      += col * sample(img)                  (if gmask_acc; needs img)
// The *_acc buffers have the accumulation type of dtype and must be initialised by the caller.
cudaError_t launch_gemm_scatter(const GeoHost &g, int dtype, int aux_dtype, const void *dense, const void *weight,
                                const void *offset, const void *mask, const void *img, void *img_grad_acc,
                                void *goff_acc, void *gmask_acc, cudaStream_t stream);

// gw_acc[d, s', tap] += sum_{b, p} dense[b, d, p] * mask * sample(img[b, s], pos)
cudaError_t launch_sample_wgrad(const GeoHost &g, int dtype, int aux_dtype, const void *dense, const void *img,
                                const void *offset, const void *mask, void *gw_acc, cudaStream_t stream);

// out[c] = sum_{b, s} x[b, c, s]; out has dtype out_dtype
cudaError_t launch_channel_sum(int dtype, int out_dtype, const void *x, int B, int C, int S, void *out,
                               cudaStream_t stream);

// dst[i] = (dst dtype) src[i]; src has the accumulation type of dst_dtype
cudaError_t launch_cast_from_acc(int dst_dtype, const void *src, void *dst, int64_t n, cudaStream_t stream);

// dst[b, c, s] = bias[c] (or 0 when bias == nullptr); dst has the accumulation type of dtype
cudaError_t launch_fill_bias(int dtype, int aux_dtype, const void *bias, int B, int C, int S, void *dst_acc,
                             cudaStream_t stream);

// ---- mask softmax (softmax.cu) -----------------------------------------------------------
cudaError_t launch_mask_softmax_fwd(int dtype, int64_t outer, int K, int64_t P, const void *in, void *out,
                                    cudaStream_t stream);
cudaError_t launch_mask_softmax_bwd(int dtype, int64_t outer, int K, int64_t P, const void *gout, const void *out,
                                    void *gin, cudaStream_t stream);

}  // namespace tvdcn_b200
