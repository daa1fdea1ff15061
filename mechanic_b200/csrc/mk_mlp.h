// mk_mlp.h — the network of the learned parts (16 -> 64 -> 64 -> 16, ReLU),
// bf16 tensor-core forward, backward and Adam on sm_100a.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace mk {
namespace mlp {

// f32 parameter layout: W1 [64][16] (column 15 = first-layer bias, input
// slot 15 is the constant 1) | W2 [64][64] | W3 [16][64] | b2 [64] | b3 [16].
constexpr uint32_t kW1 = 0, kW2 = 1024, kW3 = 5120, kWeights = 6144;
constexpr uint32_t kB2 = 6144, kB3 = 6208, kParams = 6224;
constexpr uint32_t kLossSlot = kParams;           // gradient arrays carry the loss after the parameters
constexpr uint32_t kPartialStride = 6240;         // floats per CTA partial

// Steps of one training launch: step k takes the `batch` samples from the running offset
// (from 0 again where they would pass `samples`).
constexpr uint32_t kPlanSteps = 256;
struct TrainPlan {
    uint32_t samples, batch, offset, steps;
    float lr, beta1, beta2, eps;
    float2 bias[kPlanSteps];   // per step: 1 - beta1^step, 1 - beta2^step
};

cudaError_t init(void);   // function attributes; call once outside stream capture
uint64_t scratch_bytes(uint32_t max_samples);
// y[n][y_cols] = net(x[n][16]); n from n_dev when non-null (then max_n bounds the grid).
cudaError_t forward(const float* params, const float* x, uint32_t n, const uint32_t* n_dev, uint32_t max_n, float* y,
                    uint32_t y_cols, uint32_t* error_flags, cudaStream_t s);
// Each step's gradient of (1/batch) sum_s sum_o out_w[o] (y_so - t_so)^2 and one Adam step on
// the parameters (moments m, v), its loss into losses[step].  With `grad` non-null (one step):
// the gradient into grad[kParams + 1] (loss last), and no update.
cudaError_t train(float* params, const float* x, const float* t, const float* out_w, const TrainPlan& plan, void* scratch,
                  float* grad, float* losses, float* m, float* v, uint32_t* error_flags, cudaStream_t s);

}  // namespace mlp
}  // namespace mk
