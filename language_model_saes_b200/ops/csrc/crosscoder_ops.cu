// List arithmetic of the JumpReLU crosscoder / SAE step (sm_100a).
//
// The step's codes are one list of (feature, summed pre-activation) pairs per token; every head derives from it its own codes
// (value where it passes the head's threshold theta / n_h, n_h the norm of the head's decoder row) and the terms of the
// tanh sparsity penalty  l1 * mean tanh(c * act * n_h)  (models/sparse_dictionary.py:895-905 of the reference project):
//   pen   its derivative with respect to the code, summed over the heads: the start of the shared sum's gradient d S
//   pull  its derivative with respect to n_h, summed over the tokens (per head and feature)
//   the correction of the threshold gradient at active entries (the dense window pass adds the derivative at zero activation)
// One thread per list slot walks the heads. As single tensor operations this took some twenty passes over [tokens, width]
// arrays per head, two of them scatter-adds that also sent every empty slot somewhere (crosscoder of 8 heads, 4096 tokens,
// lists 256 wide: 2.7 ms of a 22 ms step, and 55 launches per head that the host could not issue fast enough); here
// empty slots cost one load.
#include "adam.cuh"

namespace lmsae {

constexpr int JL_THREADS = 256;

__global__ void __launch_bounds__(JL_THREADS)
jumprelu_lists_kernel(const JumpReluListParams p) {
  pdl_wait();
  __shared__ float s_u[JL_THREADS / 32];
  __shared__ int s_n[JL_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long n = (long long)p.B * p.cap;
  float u_sum = 0.0f;
  int n_valid = 0;
  for (long long i = blockIdx.x * (long long)JL_THREADS + threadIdx.x; i < n; i += (long long)gridDim.x * JL_THREADS) {
    const int f = p.idx[i];
    if (f < 0) continue;  // codes and gradients of empty slots are never read
    ++n_valid;
    const float s = p.s_val[i], th = p.theta[f];
    float ds = 0.0f, dth = 0.0f;
    for (int h = 0; h < p.H; ++h) {
      const float nh = p.norm[(size_t)h * p.F + f];
      const bool active = s > __fdiv_rn(th, nh);  // (the quotient that the lists were selected against)
      p.act[(size_t)h * n + i] = active ? s : 0.0f;
      if (!active || p.coef == 0.0f) continue;
      const float x = s * nh;
      // in 64 bits: 1 - tanh^2 cancels, and the fast fp32 tanh that this file's flags select is a dozen times further off than
      // tanh rounded to fp32 (1e-4 of sech^2 at x = 3 against 8e-6)
      const double u = tanh((double)(p.stretch * x));
      const float sech2 = (float)(1.0 - u * u);
      u_sum += (float)u;
      ds += p.coef * nh * sech2;
      atomicAdd(p.pull + (size_t)h * p.F + f, p.coef * s * sech2);
      if (fabsf(x - th) < 0.5f * p.window) dth += p.coef * (sech2 - 1.0f) * (-th / p.window);
    }
    p.dS[i] = ds;
    if (dth != 0.0f) atomicAdd(p.dtheta + f, dth);
  }
  u_sum = warp_sum(u_sum);
  n_valid = __reduce_add_sync(0xffffffffu, n_valid);
  if (lane == 0) { s_u[warp] = u_sum; s_n[warp] = n_valid; }
  __syncthreads();
  if (warp == 0) {
    u_sum = warp_sum(lane < JL_THREADS / 32 ? s_u[lane] : 0.0f);
    n_valid = __reduce_add_sync(0xffffffffu, lane < JL_THREADS / 32 ? s_n[lane] : 0);
    if (lane == 0) {
      if (u_sum != 0.0f) atomicAdd(p.u_sum, u_sum);
      if (n_valid != 0) atomicAdd(p.n_valid, n_valid);
    }
  }
}

int jumprelu_lists_launch(const JumpReluListParams& p, cudaStream_t stream) {
  if (p.B <= 0 || p.cap <= 0 || p.H <= 0 || p.F <= 0) return (int)cudaErrorInvalidValue;
  const long long blocks = ((long long)p.B * p.cap + JL_THREADS - 1) / JL_THREADS;
  launch(jumprelu_lists_kernel, (int)(blocks < 148LL * 16 ? blocks : 148LL * 16), JL_THREADS, 0, stream, p);
  return (int)cudaGetLastError();
}

// What a step needs of its thresholds theta and norms: the smallest threshold theta / ||W_D,h row|| of the heads (a NaN stays one),
// and where wanted the gate by which chunk_columns_kernel finds what passes the threshold: times its gate, such a
// value is at least 1 less two roundings. Where 1 / threshold would leave the range, infinity (every positive value is looked at), below zero and for a
// NaN a NaN (everything is). (theta and the heads' summed bias are torch's: a threshold that differs
// in its last bit moves values across it.)
__global__ void __launch_bounds__(256)
jumprelu_begin_kernel(const float* __restrict__ theta, const float* __restrict__ norm, int H, int F, float* __restrict__ t_min, float* __restrict__ gate) {
  pdl_wait();
  const int f = blockIdx.x * 256 + threadIdx.x;
  if (f >= F) return;
  const float th = theta[f];
  float m = __int_as_float(0x7f800000);
  for (int h = 0; h < H; ++h) {
    const float t = __fdiv_rn(th, norm[(size_t)h * F + f]);
    if (m == m && (t != t || t < m)) m = t;
  }
  t_min[f] = m;
  if (gate != nullptr) gate[f] = m >= 0.0f ? (m > 0x1p-125f && m < 0x1p125f ? __fdiv_rn(1.0f, m) : __int_as_float(0x7f800000)) : __int_as_float(0x7fffffff);
}

int jumprelu_begin_launch(const float* theta, const float* norm, int H, int F, float* t_min, float* gate, cudaStream_t stream) {
  if (H <= 0 || F <= 0) return (int)cudaErrorInvalidValue;
  return (int)launch(jumprelu_begin_kernel, (F + 255) / 256, 256, 0, stream, theta, norm, H, F, t_min, gate);
}

// The end of a step: Adam on log theta, whose gradient is d theta * theta, and the step's figures out[0..4): loss l_rec + l_s + l_p, l_s, l_p, active entries per
// token. (As tensor operations: eight launches of a few elements.)
__global__ void __launch_bounds__(256)
jumprelu_end_kernel(const JumpReluEndParams p) {
  pdl_wait();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const float l_s = __fdiv_rn(p.l1 * *p.u_sum, p.loss_den), l_p = p.l_p != nullptr ? *p.l_p : 0.0f;
    p.out[0] = *p.l_rec + l_s + l_p;
    p.out[1] = l_s;
    p.out[2] = l_p;
    p.out[3] = __fdiv_rn((float)*p.n_valid, p.tokens);
  }
  if (p.status != nullptr && *reinterpret_cast<const volatile int*>(p.status) != 0) return;  // see sparse_grad_adam_kernel
  const int f = blockIdx.x * 256 + threadIdx.x;
  if (f >= p.F) return;
  float x = p.log_theta[f], m = p.m[f], v = p.v[f];
  adam_elem(x, m, v, p.dtheta[f] * p.theta[f], p.h);
  p.log_theta[f] = x;
  p.m[f] = m;
  p.v[f] = v;
}

int jumprelu_end_launch(const JumpReluEndParams& p, cudaStream_t stream) {
  if (p.F <= 0) return (int)cudaErrorInvalidValue;
  return (int)launch(jumprelu_end_kernel, (p.F + 255) / 256, 256, 0, stream, p);
}

}  // namespace lmsae
