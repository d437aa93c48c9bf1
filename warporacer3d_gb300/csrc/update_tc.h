// PPO's minibatch step fused on the tensor cores (update_tc.cu).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace racer {

constexpr int UPDATE_MAX_IN = 128;  // inputs a tile's shared memory holds

// Gradient partials and the samples' scalars, for one trainer.
struct UpdateWork {
  float* part = nullptr;    // [ranges][P - 2] weight gradients
  double* sums = nullptr;   // [ctas][3] log-std gradients and KL
  double* squares = nullptr;  // partial sums of grad^2
  float* samples = nullptr;   // [4][5][batch]: action 0, action 1, logp, value, advantage
  uint8_t* w1t = nullptr;     // swizzled BF16 W1^T
  int in = 0, batch = 0, ctas = 0, range = 0, ranges = 0;
};

int update_work_new(int in, int batch, UpdateWork* w);
void update_work_delete(UpdateWork* w);

// Once per update: the samples' scalars by minibatch, and W1^T from theta.
cudaError_t launch_update_begin(UpdateWork* w, int n, const float* actions, const float* logp, const float* value,
                                const float* advantage, const float* theta, cudaStream_t st);

// Where the tile kernel leaves a minibatch's activations and loss derivatives (all null: nowhere).
struct UpdateDump {
  float *h1 = nullptr, *h2 = nullptr, *o = nullptr, *d3 = nullptr;
};

// One minibatch: forward, loss, backward, gradient norm and Adam on inputs xmap (make_tmap_bf16 of [in, batch] with
// 128-row boxes), updating theta, its operand images `pack` and w->w1t; grad [P], stats (ST_NORM, ST_KL) written.
cudaError_t launch_update_minibatch(UpdateWork* w, int m, const CUtensorMap& xmap, float* theta, uint8_t* pack,
                                    float* grad, float* first, float* second, const float* c12, float* stats,
                                    const UpdateDump& dump, int* err, cudaStream_t st);

}  // namespace racer
