// The decay of a gated recurrence, exp(-rate softplus(c + bias)).
#pragma once

__device__ __forceinline__ float decay_of(float c, float rate, float bias) {
  const float z = c + bias;
  return expf(-rate * (fmaxf(z, 0.0f) + log1pf(expf(-fabsf(z)))));
}
