// Adam on one element (torch.optim.Adam without weight decay or amsgrad).
#pragma once
#include "common.cuh"
#include "kernels.h"

namespace lmsae {

__device__ __forceinline__ void adam_elem(float& p, float& m, float& v, float g, const AdamHyper& h) {
  m = h.beta1 * m + (1.0f - h.beta1) * g;
  v = h.beta2 * v + (1.0f - h.beta2) * g * g;
  const float denom = sqrtf(v) / h.bias_correction2_sqrt + h.eps;
  p -= (h.lr / h.bias_correction1) * (m / denom);
}

}  // namespace lmsae
