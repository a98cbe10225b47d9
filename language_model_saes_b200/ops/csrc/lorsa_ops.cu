// Kernels around the attention of the low-rank sparse attention step (sm_100a).
#include "adam.cuh"

namespace lmsae {

LMSAE_DEFINE_BOUNDS_FETCH(bounds_fetch_lorsa_ops)

// ---------------------------------------------------------------------------------------------
// Gradient of the pre-activations from the code gradients, and the attention backward's row statistics.
// ---------------------------------------------------------------------------------------------
// dz[t, :] is bf16(dact) at the selected heads and zero elsewhere; delta[b, h, s] = sum over the head's group of dz * z, where z is the
// code itself, so that it needs neither z nor a pass over dz. One CTA per token: the row is put together in shared memory and
// leaves in 16-byte stores, a thread per QK head adds up its group's products in slot order. Bound by writing dz:
// 2048 tokens of 8192: 33 MB. (As tensor operations: fill, scatter, three copies and the sum of a product: 130 us; here 14.)
__global__ void __launch_bounds__(256)
lorsa_dz_kernel(const int* __restrict__ idx, const float* __restrict__ act, const float* __restrict__ dact, int k, int F, int heads, int group, int seq,
                __nv_bfloat16* __restrict__ dz, float* __restrict__ delta) {
  pdl_wait();
  extern __shared__ __align__(16) uint8_t smem_raw[];
  __nv_bfloat16* row = reinterpret_cast<__nv_bfloat16*>(smem_raw);  // [F] (a multiple of 8)
  int* s_head = reinterpret_cast<int*>(row + F);                    // [k]
  float* s_prod = reinterpret_cast<float*>(s_head + k);             // [k]
  const long long t = blockIdx.x;
  for (int i = threadIdx.x; i < F / 8; i += 256) reinterpret_cast<uint4*>(row)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  for (int j = threadIdx.x; j < k; j += 256) {
    const int f = idx[t * k + j];
    s_head[j] = f >= 0 ? f / group : -1;
    if (f >= 0) {
      const __nv_bfloat16 g = __float2bfloat16(dact[t * k + j]);
      row[LMSAE_IDX(f, F)] = g;
      s_prod[j] = __bfloat162float(g) * act[t * k + j];
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < F / 8; i += 256) reinterpret_cast<uint4*>(dz + t * F)[i] = reinterpret_cast<const uint4*>(row)[i];
  const long long b = t / seq, s = t - b * seq;
  for (int h = threadIdx.x; h < heads; h += 256) {
    float d = 0.0f;
    for (int j = 0; j < k; ++j)
      if (s_head[j] == h) d += s_prod[j];
    delta[(b * heads + h) * seq + s] = d;
  }
}

int lorsa_dz_smem(int F, int k) { return F * 2 + k * 8; }

int lorsa_dz_launch(const int* idx, const float* act, const float* dact, long long tokens, int k, int F, int heads, int group, int seq,
                    __nv_bfloat16* dz, float* delta, cudaStream_t stream) {
  const int smem = lorsa_dz_smem(F, k);
  if (F % 8 != 0 || smem > 200 * 1024 || tokens > 2147483647LL) return (int)cudaErrorInvalidValue;
  if (tokens == 0) return 0;
  cudaError_t e = cudaFuncSetAttribute(lorsa_dz_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (e != cudaSuccess) return (int)e;
  launch(lorsa_dz_kernel, (int)tokens, 256, smem, stream, idx, act, dact, k, F, heads, group, seq, dz, delta);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Adam on query / key projections.
// ---------------------------------------------------------------------------------------------
// Parameters and moments are [heads, d, w] fp32, the gradient comes out of the product as [heads * w, d] and the products read bf16
// weights as [heads * w, d]: one pass per 64 x 64 tile turns the gradient on its way in and the new weights on their way out through
// shared memory. As separate passes the gradients and weights were transposed through memory (66 us for two times 3.1 M
// parameters, on top of Adam's 36). Up to two parameter sets of one shape share a launch.
// VEC: four columns a thread and access, where widths and addresses allow (3.1 M parameters twice: 51 -> 37 us).
template <bool VEC>
__global__ void __launch_bounds__(256)
adam_turned_kernel(const AdamTurnedParams p) {
  pdl_wait();
  __shared__ float tile[64][65];  // [w][d]
  if (p.status != nullptr && *reinterpret_cast<const volatile int*>(p.status) != 0) return;  // see sparse_grad_adam_kernel
  const AdamTurnedSet q = p.set[blockIdx.y];
  const int tiles_w = (p.w + 63) / 64;
  const unsigned tiles_d = (unsigned)(p.d + 63) / 64, row = blockIdx.x / tiles_d;
  const int h = (int)row / tiles_w, w0 = ((int)row - h * tiles_w) * 64, d0 = (int)(blockIdx.x - row * tiles_d) * 64;
  if constexpr (VEC) {  // (d and w are multiples of 4: whole fours are inside or outside)
    const int x = (threadIdx.x & 15) * 4, y0 = threadIdx.x >> 4;
#pragma unroll
    for (int y = y0; y < 64; y += 16) {
      if (w0 + y < p.w && d0 + x < p.d) {
        const float4 g = __ldcs(reinterpret_cast<const float4*>(q.g + ((size_t)h * p.w + w0 + y) * p.d + d0 + x));
        tile[y][x] = g.x; tile[y][x + 1] = g.y; tile[y][x + 2] = g.z; tile[y][x + 3] = g.w;
      }
    }
    float4 pp[4], pm[4], pv[4];  // (all of a thread's loads before the first is used)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int y = y0 + i * 16;
      if (d0 + y < p.d && w0 + x < p.w) {
        const size_t o = ((size_t)h * p.d + d0 + y) * p.w + w0 + x;
        pp[i] = *reinterpret_cast<const float4*>(q.p + o);
        pm[i] = *reinterpret_cast<const float4*>(q.m + o);
        pv[i] = *reinterpret_cast<const float4*>(q.v + o);
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int y = y0 + i * 16;
      if (d0 + y < p.d && w0 + x < p.w) {
        const size_t o = ((size_t)h * p.d + d0 + y) * p.w + w0 + x;
        adam_elem(pp[i].x, pm[i].x, pv[i].x, tile[x][y], p.h); adam_elem(pp[i].y, pm[i].y, pv[i].y, tile[x + 1][y], p.h);
        adam_elem(pp[i].z, pm[i].z, pv[i].z, tile[x + 2][y], p.h); adam_elem(pp[i].w, pm[i].w, pv[i].w, tile[x + 3][y], p.h);
        *reinterpret_cast<float4*>(q.p + o) = pp[i];
        *reinterpret_cast<float4*>(q.m + o) = pm[i];
        *reinterpret_cast<float4*>(q.v + o) = pv[i];
        tile[x][y] = pp[i].x; tile[x + 1][y] = pp[i].y; tile[x + 2][y] = pp[i].z; tile[x + 3][y] = pp[i].w;
      }
    }
    __syncthreads();
#pragma unroll
    for (int y = y0; y < 64; y += 16) {
      if (w0 + y < p.w && d0 + x < p.d)
        *reinterpret_cast<uint2*>(q.shadow + ((size_t)h * p.w + w0 + y) * p.d + d0 + x) =
            make_uint2(pack_bf16x2(tile[y][x], tile[y][x + 1]), pack_bf16x2(tile[y][x + 2], tile[y][x + 3]));
    }
    return;
  }
  const int x = threadIdx.x & 63, y0 = threadIdx.x >> 6;
#pragma unroll 4
  for (int y = y0; y < 64; y += 4)
    if (w0 + y < p.w && d0 + x < p.d) tile[y][x] = __ldcs(q.g + ((size_t)h * p.w + w0 + y) * p.d + d0 + x);
  __syncthreads();
#pragma unroll 4
  for (int y = y0; y < 64; y += 4) {
    if (d0 + y >= p.d || w0 + x >= p.w) continue;
    const size_t o = ((size_t)h * p.d + d0 + y) * p.w + w0 + x;
    float pi = q.p[o], mi = q.m[o], vi = q.v[o];
    adam_elem(pi, mi, vi, tile[x][y], p.h);
    q.p[o] = pi;
    q.m[o] = mi;
    q.v[o] = vi;
    tile[x][y] = pi;
  }
  __syncthreads();
#pragma unroll 4
  for (int y = y0; y < 64; y += 4)
    if (w0 + y < p.w && d0 + x < p.d) q.shadow[((size_t)h * p.w + w0 + y) * p.d + d0 + x] = __float2bfloat16(tile[y][x]);
}

int adam_turned_launch(const AdamTurnedParams& p, int n_sets, cudaStream_t stream) {
  if (n_sets < 1 || n_sets > 2 || p.heads <= 0 || p.d <= 0 || p.w <= 0) return (int)cudaErrorInvalidValue;
  const long long tiles = (long long)p.heads * ((p.w + 63) / 64) * ((p.d + 63) / 64);
  if (tiles > 2147483647LL) return (int)cudaErrorInvalidValue;
  bool vec = p.d % 4 == 0 && p.w % 4 == 0;
  for (int i = 0; i < n_sets; ++i)
    vec = vec && ((reinterpret_cast<uintptr_t>(p.set[i].p) | reinterpret_cast<uintptr_t>(p.set[i].m) | reinterpret_cast<uintptr_t>(p.set[i].v) |
                   reinterpret_cast<uintptr_t>(p.set[i].g) | reinterpret_cast<uintptr_t>(p.set[i].shadow)) % 16 == 0);
  auto kern = vec ? adam_turned_kernel<true> : adam_turned_kernel<false>;
  launch(kern, dim3((unsigned)tiles, n_sets), 256, 0, stream, p);
  return (int)cudaGetLastError();
}

}  // namespace lmsae
