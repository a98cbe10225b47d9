// Cross-layer transcoder decoder fan-out on sparse codes (sm_100a, SIMT gather kernels: HBM/L2-bound).
//
// A cross-layer transcoder decodes the features of source layer s into every target layer t >= s:
//   y[t, b, :] = b_D[t] + sum_{s <= t} sum_f a[b, s, f] * W_D[t][s, f, :]
// (models/clt.py:629-709 of the reference project, which runs one dense or CSR product per (s, t) pair and one
// all-reduce per target layer). Here the codes of a token are one padded list of (c = s * F + f, value) pairs, and
//
//   clt_decode_kernel   warps of a (token, target layer) gather the rows W_D[t][s, f, :] of that token's codes with
//                       s <= t and accumulate them in registers: every target layer in one launch, no dense product;
//   clt_dact_kernel     d a[b, j] = sum_{t >= s} d y[t, b, :] . W_D[t][s, f, :]   (one CTA per token, a warp per code);
//   clt_wgrad_kernel    d W_D[t][s, f, :] = sum_{b in rows(c)} a[b, c] * d y[t, b, :] for every t >= s from the
//                       by-feature lists of a counting sort: one CTA per active (s, f), no atomics; rows of features
//                       that did not fire are not touched (the caller hands in zero-filled gradients).
//
// W_D[t] is its own allocation of shape [t + 1, F, d] (bf16); the kernels take the table of base pointers by value.
#include "gather.cuh"
#include "kernels.h"

namespace lmsae {

LMSAE_DEFINE_BOUNDS_FETCH(bounds_fetch_clt_ops)

// ---------------------------------------------------------------------------------------------
// forward
// ---------------------------------------------------------------------------------------------
// One warp per (target layer, token, segment of 256 columns), ordered by target layer: all tokens of a layer are resident at
// once and walk their lists, which are ordered by source layer, in step, so that the rows gathered at any time come from a
// few [F, d] slices of W_D[t] that fit the L2 cache. One CTA per token and layer, token by token, read every slice from
// HBM again for almost every row: 3.29 ms against 1.54 ms here (12 layers x 24576 features, d 768, 2048 tokens, k 64 per layer:
// 15.7 GB of rows, 10.2 TB/s).
constexpr int CLT_DEC_WARPS = 8;

__global__ void __launch_bounds__(CLT_DEC_WARPS * 32)
clt_decode_kernel(const CltTable tab, const int* __restrict__ idx, const float* __restrict__ val, int B, int K, int L,
                  int F, int d, int nseg, const float* __restrict__ bias, float* __restrict__ out_f32,
                  __nv_bfloat16* __restrict__ out_bf16) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int nvec = d / 8;
  const long long item = (long long)blockIdx.x * CLT_DEC_WARPS + (threadIdx.x >> 5);
  const long long per_layer = (long long)B * nseg;
  if (item >= per_layer * L) return;
  const int layer_rank = (int)(item / per_layer);
  const int t = L - 1 - layer_rank;  // deepest target (longest lists) first
  const long long rest = item - (long long)layer_rank * per_layer;
  const int row = (int)(rest / nseg), seg = (int)(rest - (long long)row * nseg);
  const int v[1] = {seg * 32 + lane};
  const bool in[1] = {v[0] < nvec};
  float acc[1][8];
  const long long limit = (long long)(t + 1) * F;  // codes c < limit come from source layers s <= t
  gather_rows_warp<1>(idx + (size_t)row * K, val + (size_t)row * K, K, tab.W[t], d, limit, limit, v, in, acc);
  if (!in[0]) return;
  const int c0 = v[0] * 8;
  const size_t obase = ((size_t)t * B + row) * d;
  if (bias != nullptr) {
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[0][i] += bias[(size_t)t * d + c0 + i];
  }
  if (out_f32 != nullptr) {
    float4* o = reinterpret_cast<float4*>(out_f32 + obase + c0);
    o[0] = make_float4(acc[0][0], acc[0][1], acc[0][2], acc[0][3]);
    o[1] = make_float4(acc[0][4], acc[0][5], acc[0][6], acc[0][7]);
  }
  if (out_bf16 != nullptr) {
    uint4 o;
    o.x = pack_bf16x2(acc[0][0], acc[0][1]);
    o.y = pack_bf16x2(acc[0][2], acc[0][3]);
    o.z = pack_bf16x2(acc[0][4], acc[0][5]);
    o.w = pack_bf16x2(acc[0][6], acc[0][7]);
    *reinterpret_cast<uint4*>(out_bf16 + obase + c0) = o;
  }
}

int clt_decode_launch(const CltTable& tab, const int* idx, const float* val, int B, int K, int L, int F, int d,
                      const float* bias, float* out_f32, __nv_bfloat16* out_bf16, cudaStream_t stream) {
  if (d % 8 != 0 || d > 8192 || L < 1 || L > kMaxCltLayers) return (int)cudaErrorInvalidValue;
  if ((long long)L * F > 2147483647LL) return (int)cudaErrorInvalidValue;
  if (B <= 0) return 0;
  const int nseg = (d / 8 + 31) / 32;
  const long long blocks = ((long long)B * L * nseg + CLT_DEC_WARPS - 1) / CLT_DEC_WARPS;
  if (blocks > 2147483647LL) return (int)cudaErrorInvalidValue;
  launch(clt_decode_kernel, (int)blocks, CLT_DEC_WARPS * 32, 0, stream, tab, idx, val, B, K, L, F, d, nseg, bias, out_f32, out_bf16);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// gradient of the codes
// ---------------------------------------------------------------------------------------------
constexpr int CLT_DACT_THREADS = 256;

__global__ void __launch_bounds__(CLT_DACT_THREADS)
clt_dact_kernel(const CltTable tab, const int* __restrict__ idx, int B, int K, int L, int F, int d,
                const __nv_bfloat16* __restrict__ dy, float* __restrict__ dval) {
  extern __shared__ uint8_t smem_raw[];
  float* s_dy = reinterpret_cast<float*>(smem_raw);          // [d]
  float* s_acc = s_dy + d;                                   // [K]
  int* s_idx = reinterpret_cast<int*>(s_acc + K);            // [K]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = d / 8;
  for (int row = blockIdx.x; row < B; row += gridDim.x) {
    __syncthreads();
    for (int j = threadIdx.x; j < K; j += CLT_DACT_THREADS) {
      s_idx[j] = idx[(size_t)row * K + j];
      s_acc[j] = 0.0f;
    }
    __syncthreads();
    for (int t = 0; t < L; ++t) {
      const long long limit = (long long)(t + 1) * F;
      __syncthreads();
      for (int v = threadIdx.x; v < nvec; v += CLT_DACT_THREADS) {
        float f[8];
        bf16x8_to_float(__ldg(reinterpret_cast<const uint4*>(dy + ((size_t)t * B + row) * d) + v), f);
#pragma unroll
        for (int i = 0; i < 8; ++i) s_dy[v * 8 + i] = f[i];
      }
      __syncthreads();
      const __nv_bfloat16* Wt = tab.W[t];
      // code j always belongs to warp j % 8, so its accumulator has one writer
      for (int j = warp; j < K; j += CLT_DACT_THREADS / 32) {
        const int c = s_idx[j];
        if (c < 0 || c >= limit) continue;
        const uint4* wrow = reinterpret_cast<const uint4*>(Wt + (size_t)c * d);
        float dot = 0.0f;
        for (int v = lane; v < nvec; v += 32) {
          float wv[8];
          bf16x8_to_float(__ldg(wrow + v), wv);
          const float* g = s_dy + v * 8;
#pragma unroll
          for (int i = 0; i < 8; ++i) dot = fmaf(wv[i], g[i], dot);
        }
        dot = warp_sum(dot);
        if (lane == 0) s_acc[j] += dot;
      }
    }
    __syncthreads();
    for (int j = threadIdx.x; j < K; j += CLT_DACT_THREADS) dval[(size_t)row * K + j] = s_acc[j];
  }
}

int clt_dact_launch(const CltTable& tab, const int* idx, int B, int K, int L, int F, int d, const __nv_bfloat16* dy,
                    float* dval, cudaStream_t stream) {
  if (d % 8 != 0 || L < 1 || L > kMaxCltLayers) return (int)cudaErrorInvalidValue;
  const size_t smem = (size_t)d * 4 + (size_t)K * 8;
  if (smem > 160 * 1024) return (int)cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(clt_dact_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
  if (e != cudaSuccess) return (int)e;
  if (B <= 0) return 0;
  const int blocks = B < 148 * 8 ? B : 148 * 8;
  launch_plain(clt_dact_kernel, blocks, CLT_DACT_THREADS, smem, stream, tab, idx, B, K, L, F, d, dy, dval);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// gradient of the decoders
// ---------------------------------------------------------------------------------------------
constexpr int CLT_WG_THREADS = 256;

__global__ void __launch_bounds__(CLT_WG_THREADS)
clt_wgrad_kernel(const CltGradTable tab, const int* __restrict__ offsets, const int* __restrict__ entries,
                 const float* __restrict__ act, int B, int K, int L, int F, int d,
                 const __nv_bfloat16* __restrict__ dy) {
  const long long n_codes = (long long)L * F;
  for (long long c = blockIdx.x; c < n_codes; c += gridDim.x) {
    const int e0 = offsets[c], e1 = offsets[c + 1];
    if (e0 == e1) continue;
    const int s = (int)(c / F);
    for (int t = s; t < L; ++t) {
      float* grow = tab.G[t] + (size_t)c * d;
      const __nv_bfloat16* dyt = dy + (size_t)t * B * d;
      for (int c0 = threadIdx.x * 4; c0 < d; c0 += CLT_WG_THREADS * 4) {
        float g[4] = {0.f, 0.f, 0.f, 0.f};
        for (int e = e0; e < e1; ++e) {
          const int ent = entries[e];
          const int row = ent / K;
          const float a = act[ent];
          const uint2 u = __ldg(reinterpret_cast<const uint2*>(dyt + (size_t)row * d + c0));
          const float2 d01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
          const float2 d23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
          g[0] = fmaf(a, d01.x, g[0]); g[1] = fmaf(a, d01.y, g[1]);
          g[2] = fmaf(a, d23.x, g[2]); g[3] = fmaf(a, d23.y, g[3]);
        }
        *reinterpret_cast<float4*>(grow + c0) = make_float4(g[0], g[1], g[2], g[3]);
      }
    }
  }
}

int clt_wgrad_launch(const CltGradTable& tab, const int* offsets, const int* entries, const float* act, int B, int K,
                     int L, int F, int d, const __nv_bfloat16* dy, cudaStream_t stream) {
  if (d % 4 != 0 || L < 1 || L > kMaxCltLayers) return (int)cudaErrorInvalidValue;
  const long long n_codes = (long long)L * F;
  if (n_codes <= 0 || n_codes > 2147483647LL) return (int)cudaErrorInvalidValue;
  const int blocks = (int)(n_codes < 148LL * 16 ? n_codes : 148LL * 16);
  launch_plain(clt_wgrad_kernel, blocks, CLT_WG_THREADS, 0, stream, tab, offsets, entries, act, B, K, L, F, d, dy);
  return (int)cudaGetLastError();
}

}  // namespace lmsae
