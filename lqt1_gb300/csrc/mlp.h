// mlp.h -- the learned surrogate's network (48 -> 128 -> 128 -> 48, SiLU).
//
// Inputs (48): the 38 evolving states of a cell (V, 8 concentrations, the 29
// gates/fluxes that change) and 6 parameters (GKs, PCa and GKs-ISO factors of
// the cell's model, endo/epi/M one-hot), normalised per feature, zero padded.
// Outputs (48): the normalised correction of the 38 states over one macro step
// (nsub plain steps minus one coarse step) without diffusion or stimulus, zero
// padded.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace lqt {

constexpr int kMlpIn = 48, kMlpHid = 128, kMlpOut = 48;
constexpr int kMlpNState = 38, kMlpNParam = 6;

// Device view of the network: weights stored [out][in] row-major (BF16), biases FP32.
struct MlpDev {
    const __nv_bfloat16 *w1t, *w2t, *w3t;   // [128][48], [128][128], [48][128]
    const float *b1, *b2, *b3;              // [128], [128], [48]
    const float *w2f, *w3f;                 // FP32 master copies of W2, W3
};

}  // namespace lqt
struct lqt_mlp;
namespace lqt {
// Device weights and normalisation (in_mean, in_scale, out_scale) of a network.
bool mlp_device_view(const lqt_mlp *m, MlpDev *w, const float **norm);

cudaError_t launch_mlp_infer_tc(const __nv_bfloat16 *X, float *Y, const MlpDev &w, int64_t n, int *err, int swap,
                                cudaStream_t st);

// Training (k_mlp_train.cu): gradient slices of a batch, one per CTA
// (mlp_grad_slices of them, kMlpNParam32 floats each, and one loss sum each)
// and the row gradients (kMlpNBias values a row); and their ordered sums with,
// for lr > 0, one Adam step.
constexpr int kMlpNParam32 = 2 * kMlpIn * kMlpHid + kMlpHid * kMlpHid + 2 * kMlpHid + kMlpOut;
constexpr int kMlpNBias = 2 * kMlpHid + kMlpOut;
int mlp_grad_slices(int64_t B);
cudaError_t launch_mlp_grad(const __nv_bfloat16 *X, const float *T, int64_t B, int nvalid, const MlpDev &w, float *part,
                            double *lossp, __nv_bfloat16 *grow, int *err, cudaStream_t st);
cudaError_t launch_mlp_update(const float *part, const double *lossp, int slices, const __nv_bfloat16 *grow, int64_t B,
                              float *g, double *loss, float *p, float *m, float *v, __nv_bfloat16 *pb, float lr, float b1,
                              float b2, float eps, float c1, float c2, cudaStream_t st);

}  // namespace lqt
