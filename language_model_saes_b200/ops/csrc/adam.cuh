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

// The same with the factors worked out once, for the kernels that stream rows of parameters.
struct AdamConst {
  float b1, b2, c1, c2, inv_bc2, step, eps;
};

__device__ __forceinline__ void adam_update(float& p, float& m, float& v, float g, const AdamConst& h) {
  m = fmaf(h.b1, m, h.c1 * g);
  v = fmaf(h.b2, v, h.c2 * g * g);
  p = fmaf(-h.step, m / fmaf(sqrtf(v), h.inv_bc2, h.eps), p);
}

// One row of a parameter or moment matrix to shared memory, on a bulk copy.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Whether a feature has more than n entries, the same in every thread of the CTA (a barrier).
__device__ __forceinline__ bool any_longer_list(const GradAdamParams& p, int n) {
  bool any = false;
  for (int i = threadIdx.x, n_heavy = p.heavy[0]; i < n_heavy; i += blockDim.x) {
    const int f = p.heavy[1 + i] - p.heavy_base;
    any |= f >= 0 && f < p.F && p.offsets[f + 1] - p.offsets[f] > n;
  }
  return __syncthreads_or(any) != 0;
}

}  // namespace lmsae
