// PPO's loss derivatives for one sample (racer/ppo.mojo:242-250, 276-304),
// shared by the loss kernel and the fused minibatch: both translation units
// are built with --fmad=false, so either gives the same bits.
#pragma once
#include "common.cuh"
#include "rmath.h"

namespace racer {
namespace {

// racer/ppo.mojo:249-250 from the device-side sums of the advantages and their squares.
__device__ __forceinline__ void advantage_moments(const float* moments, int batch, float* mean, float* scale) {
  const float samples = (float)((long)batch * MINIBATCHES);
  *mean = moments[0] / samples;
  const float var = moments[1] / samples - *mean * *mean;
  *scale = 1.0f / sqrtf(fmaxf(var, 1e-8f));
}

// d[0..2] = the derivatives by the three outputs, d[3..4] by the log standard deviations, d[5] = the KL estimate's
// term. ls = log std, invvar = exp(-2 ls).
__device__ __forceinline__ void ppo_loss(float action0, float action1, float logp, float value, float advantage,
                                         float o0, float o1, float o2, const float* ls, const float* invvar,
                                         float adv_mean, float adv_scale, float batch, float* d) {
  const float error[2] = {action0 - o0, action1 - o1};
  float new_logp = 0.0f;
#pragma unroll
  for (int a = 0; a < 2; ++a) new_logp -= (((0.5f * error[a]) * error[a]) * invvar[a] + ls[a]) + HALF_LOG_2PI;
  const float logratio = new_logp - logp;
  const float ratio = rmath::expf_(logratio);
  const float a_hat = (advantage - adv_mean) * adv_scale;
  float dlogp = (-a_hat * ratio) / batch;
  if ((a_hat >= 0.0f && ratio > 1.0f + CLIP) || (a_hat < 0.0f && ratio < 1.0f - CLIP)) dlogp = 0.0f;
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    d[a] = (dlogp * error[a]) * invvar[a];
    d[OUT + a] = dlogp * ((error[a] * error[a]) * invvar[a] - 1.0f);
  }
  const float e = (o2 - value) - advantage;
  d[2] = (0.5f * fminf(fmaxf(e, -1.0f), 1.0f)) / batch;
  d[OUT + 2] = (ratio - 1.0f) - logratio;
}

}  // namespace
}  // namespace racer
