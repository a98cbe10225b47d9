// acts [B, F] (dense fp32 storage of sparse activations) times W [F, d] in fp32: the decoder of inference (sm_100a).
//
// A product of 4096 x 24576 x 768 takes 3.1 ms on the fp32 pipes, nearly all of it multiplications by zero. Here a CTA takes one
// token: its eight warps compact the non-zeros of an eighth of the row each into shared memory (in column order: sums do not depend
// on timing), the lists are joined, and all threads then add up the gathered rows of W, eight on their way at once. Bound by reading acts once (HBM)
// and the rows of W (L2); 4096 x 24576 x 768 with 50 non-zeros a row, with the bias:
// 3073 us as a product and a sum, 138 with W looked through by itself, the lists one after the other and the bias in a launch of its own, 118 here.
//
// Results are those of the dense product also where skipping a zero is not allowed or does not pay: with a W that holds an infinity or
// a NaN (0 * inf is NaN) all rows, and else rows with more than `most` non-zeros, or more than kWarpList in an eighth, are
// left to rows_product.cu, which leaves at once where there are none. The decision is taken on the device: the host waits for nothing. W is looked
// through by the launch's first CTAs while the others gather (by itself: 20 us); where something is found, what they gathered is written over.
#include "gather.cuh"
#include "kernels.h"

namespace lmsae {

LMSAE_DEFINE_BOUNDS_FETCH(bounds_fetch_dense_decode)

namespace {

constexpr int DD_THREADS = 256;
constexpr int kWarpList = 256;

// Whether w holds an infinity or a NaN: this CTA's share of `ctas`.
__device__ __forceinline__ void look_through(const float* __restrict__ w, long long n, int ctas, int* __restrict__ found) {
  bool bad = false;
  const long long n4 = n / 4, stride = (long long)ctas * DD_THREADS;
#pragma unroll 8
  for (long long i = blockIdx.x * (long long)DD_THREADS + threadIdx.x; i < n4; i += stride) {
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(w) + i);
    bad |= (u.x & 0x7f800000u) == 0x7f800000u || (u.y & 0x7f800000u) == 0x7f800000u || (u.z & 0x7f800000u) == 0x7f800000u ||
           (u.w & 0x7f800000u) == 0x7f800000u;
  }
  if (bad) *found = 1;
}

__global__ void __launch_bounds__(DD_THREADS, 5)
sparse_rows_kernel(const float* __restrict__ acts, const float* __restrict__ W, const float* __restrict__ bias, int F, int d, int most, int lookers, int B,
                   int* __restrict__ todo, float* __restrict__ out) {
  pdl_wait();
  __shared__ int s_idx[8][kWarpList], s_all_idx[8 * kWarpList];
  __shared__ float s_val[8][kWarpList], s_all_val[8 * kWarpList];
  __shared__ int s_n[8];
  __shared__ float4 s_part[DD_THREADS];
  if ((int)blockIdx.x < lookers) {
    look_through(W, (long long)F * d, lookers, todo + 1 + B);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = (int)blockIdx.x - lookers;
  const uint4* a = reinterpret_cast<const uint4*>(acts + (size_t)row * F);
  const int nv = F / 4, per = (nv + 7) / 8, v0 = min(nv, warp * per), v1 = min(nv, v0 + per);
  int n = 0;
  for (int v = v0; v < v1; v += 128) {
    uint4 u[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int at = v + i * 32 + lane;
      u[i] = at < v1 ? __ldcs(a + at) : make_uint4(0u, 0u, 0u, 0u);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t x[4] = {u[i].x, u[i].y, u[i].z, u[i].w};
      unsigned m = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) m |= (unsigned)((x[e] & 0x7fffffffu) != 0u) << e;
      if (__ballot_sync(0xffffffffu, m != 0u) == 0u) continue;
      int inc = __popc(m);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      int slot = n + inc - __popc(m);
      n += __shfl_sync(0xffffffffu, inc, 31);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if ((m >> e) & 1u) {
          if (slot < kWarpList) {
            s_idx[warp][slot] = (v + i * 32 + lane) * 4 + e;
            s_val[warp][slot] = __uint_as_float(x[e]);
          }
          ++slot;
        }
      }
    }
  }
  if (lane == 0) s_n[warp] = n;
  __syncthreads();
  bool over = false;
  int all = 0, before = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) {
    over |= s_n[w] > kWarpList;
    before += w < warp ? s_n[w] : 0;
    all += s_n[w];
  }
  if (over || all > most) {
    if (threadIdx.x == 0) todo[1 + atomicAdd(todo, 1)] = row;
    return;
  }
  for (int e = lane; e < n; e += 32) {
    s_all_idx[before + e] = s_idx[warp][e];
    s_all_val[before + e] = s_val[warp][e];
  }
  __syncthreads();
  // four columns a thread; with few columns several groups of threads share the entries and add up in a fixed order
  const int cols = d / 4, groups = cols >= DD_THREADS ? 1 : DD_THREADS / cols;
  const int g = groups == 1 ? 0 : (int)threadIdx.x / cols;
  for (int c = groups == 1 ? (int)threadIdx.x : (int)threadIdx.x % cols; c < cols; c += DD_THREADS) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    if (g < groups) {
      const float4* Wc = reinterpret_cast<const float4*>(W) + c;
      constexpr int U = 8;
      for (int e = g; e < all; e += U * groups) {
        float4 r[U];
        float f[U];
#pragma unroll
        for (int i = 0; i < U; ++i) {
          const int at = e + i * groups;
          f[i] = at < all ? s_all_val[at] : 0.0f;
          r[i] = at < all ? __ldg(Wc + (size_t)LMSAE_IDX(s_all_idx[at], F) * cols) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < U; ++i) {
          fma2(acc.x, acc.y, r[i].x, r[i].y, f[i], f[i]);
          fma2(acc.z, acc.w, r[i].z, r[i].w, f[i], f[i]);
        }
      }
    }
    if (groups > 1) {  // (one pass of the loop for every thread: cols < DD_THREADS)
      s_part[threadIdx.x] = acc;
      __syncthreads();
      if (g != 0) break;
      for (int q = 1; q < groups; ++q) {
        const float4 o = s_part[q * cols + c];
        acc.x += o.x; acc.y += o.y; acc.z += o.z; acc.w += o.w;
      }
    }
    if (bias != nullptr) {
      const float4 o = __ldg(reinterpret_cast<const float4*>(bias) + c);
      acc.x += o.x; acc.y += o.y; acc.z += o.z; acc.w += o.w;
    }
    reinterpret_cast<float4*>(out + (size_t)row * d)[c] = acc;
  }
}

}  // namespace

// todo: int [2 + B + part_tiles], zeroed by the caller: how many rows are left to the product, which, whether W holds an infinity or a
// NaN, and the product's counters. most: non-zeros up to which a row is gathered. F % 4 == 0, d % 4 == 0, pointers 16-byte aligned.
int dense_decode_launch(const float* acts, const float* W, const float* bias, int B, int F, int d, int most, int* todo, float* part, long long part_floats, int part_tiles,
                        float* out, cudaStream_t stream) {
  const uintptr_t align = reinterpret_cast<uintptr_t>(acts) | reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(bias);
  if (F % 4 != 0 || d % 4 != 0 || align % 16 != 0 || F <= 0 || d <= 0) return (int)cudaErrorInvalidValue;
  if (B <= 0) return 0;
  const long long n = (long long)F * d;
  const long long blocks = (n / 4 + DD_THREADS * 8 - 1) / (DD_THREADS * 8);
  // one of an SM's five CTAs looks through W beside the rows of acts, three where W is the longer of the two: by themselves 148 CTAs read 3.6 TB/s
  // (256 x 131072 x 4096 with 50 non-zeros a row: 595 -> 396 us, 512 x 65536 x 2048: 191 -> 153; 4096 x 24576 x 768: 130, with three 132)
  const int most_lookers = 148 * (d > B ? 3 : 1), lookers = (int)(blocks < most_lookers ? blocks : most_lookers);
  if (B > 2147483647 - lookers) return (int)cudaErrorInvalidValue;
  const cudaError_t e = launch(sparse_rows_kernel, lookers + B, DD_THREADS, 0, stream, acts, W, bias, F, d, most, lookers, B, todo, out);
  if (e != cudaSuccess) return (int)e;
  RowsProductParams r = {};
  r.A = acts; r.B = W; r.C = out; r.N = d; r.K = F; r.rows = todo; r.max_rows = B; r.every = todo + 1 + B; r.bias = bias;
  r.part = part; r.part_floats = part_floats; r.part_done = todo + 2 + B; r.part_tiles = part_tiles;
  return rows_product_launch(r, true, stream);
}

}  // namespace lmsae
