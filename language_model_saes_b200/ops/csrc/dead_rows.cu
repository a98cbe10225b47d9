// Dead features of an Aux-K step and the compact dictionary of their rows (sm_100a).
//
// From the fire counts of a step: every feature's number of tokens since it last fired, which features are dead by that, and the rows of the first
// `cap` of them (ascending; alive ones behind them with a gate of 0 and rows of zeros), their biases and gates, and every feature's row in the
// compact dictionary. As tensor operations (comparisons, sums, a sort of flags, four gathers, a scatter) these were some twenty-five launches, 100 us
// of a step of 3.4 ms; three launches here. Bound by the copies of the rows (9216 rows of 2048, twice 38 MB in and out).
#include "common.cuh"
#include "kernels.h"

namespace lmsae {

namespace {
constexpr int DR_THREADS = 256, DR_PER = 4, DR_BLOCK = DR_THREADS * DR_PER;  // features per CTA

// Exclusive prefix of `mine` over the CTA; the sum in `total`.
__device__ __forceinline__ int cta_prefix(int mine, int (&words)[DR_THREADS / 32], int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int sum = mine;
#pragma unroll
  for (int o = 1; o < 32; o *= 2) {
    const int v = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= o) sum += v;
  }
  if (lane == 31) words[warp] = sum;
  __syncthreads();
  int before = sum - mine;
  total = 0;
#pragma unroll
  for (int w = 0; w < DR_THREADS / 32; ++w) {
    if (w < warp) before += words[w];
    total += words[w];
  }
  __syncthreads();
  return before;
}
}  // namespace

__global__ void __launch_bounds__(DR_THREADS)
dead_count_kernel(const int* __restrict__ fired, const long long* __restrict__ since, const long long* __restrict__ n_valid, long long threshold, int F,
                  long long* __restrict__ since_out, uint8_t* __restrict__ is_dead, int* __restrict__ block_count) {
  pdl_wait();
  const long long n = *n_valid;
  int mine = 0;
#pragma unroll
  for (int i = 0; i < DR_PER; ++i) {
    const int f = blockIdx.x * DR_BLOCK + i * DR_THREADS + (int)threadIdx.x;
    if (f >= F) continue;
    const long long s = fired[f] > 0 ? 0 : since[f] + n;
    since_out[f] = s;
    is_dead[f] = s >= threshold;
    mine += s >= threshold;
  }
  __shared__ int words[DR_THREADS / 32];
  int total;
  cta_prefix(mine, words, total);
  if (threadIdx.x == 0) block_count[blockIdx.x] = total;
}

__global__ void __launch_bounds__(DR_THREADS)
dead_rows_kernel(const DeadRowsParams p) {
  pdl_wait();
  __shared__ int words[DR_THREADS / 32];
  int before = 0, all = 0;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += DR_THREADS) {
    const int n = p.block_count[b];
    all += n;
    if (b < (int)blockIdx.x) before += n;
  }
  int n_dead, first;
  cta_prefix(all, words, n_dead);
  cta_prefix(before, words, first);
  // a thread's features lie beside one another here, so that ranks ascend with them
  const int f0 = blockIdx.x * DR_BLOCK + (int)threadIdx.x * DR_PER;
  bool dead[DR_PER];
  int mine = 0, total;
#pragma unroll
  for (int i = 0; i < DR_PER; ++i) {
    dead[i] = f0 + i < p.F && p.is_dead[f0 + i] != 0;
    mine += dead[i];
  }
  int rank = first + cta_prefix(mine, words, total);  // dead features before this one
#pragma unroll
  for (int i = 0; i < DR_PER; ++i) {
    const int f = f0 + i;
    if (f >= p.F) break;
    const int slot = dead[i] ? rank : n_dead + (f - rank);
    if (slot < p.cap) {
      p.order[slot] = f;
      p.bias_out[slot] = p.bias[f];
      p.gate_out[slot] = !dead[i] ? 0.0f : p.gate != nullptr ? p.gate[f] : 1.0f;
    }
    p.row_of[f] = dead[i] && rank < p.cap ? rank : -1;
    rank += dead[i];
  }
  if (blockIdx.x == 0) {
    for (int s = p.F + (int)threadIdx.x; s < p.cap; s += DR_THREADS) {  // (a capacity rounded up beyond the features)
      p.order[s] = 0;
      p.bias_out[s] = p.bias[0];
      p.gate_out[s] = 0.0f;
    }
    if (threadIdx.x == 0) {
      *p.n_dead = n_dead;
      *p.any = n_dead > 0 ? 1.0f : 0.0f;
      if (n_dead > p.capacity) *p.truncated += 1;
    }
  }
}

// Rows order[r] of two matrices of 16-byte vectors; zeros from row n_dead on.
__global__ void __launch_bounds__(DR_THREADS)
dead_gather_kernel(const int* __restrict__ order, const long long* __restrict__ n_dead, int cap, int vecs, const uint4* __restrict__ a, const uint4* __restrict__ b,
                   uint4* __restrict__ a_out, uint4* __restrict__ b_out) {
  pdl_wait();
  const int n = (int)min((long long)cap, *n_dead);
  for (int r = blockIdx.x; r < cap; r += gridDim.x) {
    const size_t from = (size_t)(r < n ? order[r] : 0) * vecs, to = (size_t)r * vecs;
    for (int v = threadIdx.x; v < 2 * vecs; v += DR_THREADS) {
      const int i = v < vecs ? v : v - vecs;
      const uint4 x = r < n ? __ldg((v < vecs ? a : b) + from + i) : make_uint4(0u, 0u, 0u, 0u);
      (v < vecs ? a_out : b_out)[to + i] = x;
    }
  }
}

int dead_rows_blocks(int F) { return (F + DR_BLOCK - 1) / DR_BLOCK; }

int dead_rows_launch(const DeadRowsParams& p, const int* fired, const long long* since, const long long* n_valid, long long threshold, long long* since_out,
                     const __nv_bfloat16* WE, const __nv_bfloat16* WD, int d, __nv_bfloat16* we_out, __nv_bfloat16* wd_out, cudaStream_t stream) {
  if (p.F <= 0 || p.cap <= 0 || d <= 0 || d % 8 != 0 ||
      ((reinterpret_cast<uintptr_t>(WE) | reinterpret_cast<uintptr_t>(WD) | reinterpret_cast<uintptr_t>(we_out) | reinterpret_cast<uintptr_t>(wd_out)) & 15) != 0)
    return (int)cudaErrorInvalidValue;
  const int blocks = dead_rows_blocks(p.F);
  launch(dead_count_kernel, blocks, DR_THREADS, 0, stream, fired, since, n_valid, threshold, p.F, since_out, p.is_dead, p.block_count);
  launch(dead_rows_kernel, blocks, DR_THREADS, 0, stream, p);
  launch(dead_gather_kernel, p.cap < 148 * 8 ? p.cap : 148 * 8, DR_THREADS, 0, stream, p.order, p.n_dead, p.cap, d / 8, reinterpret_cast<const uint4*>(WE),
         reinterpret_cast<const uint4*>(WD), reinterpret_cast<uint4*>(we_out), reinterpret_cast<uint4*>(wd_out));
  return (int)cudaGetLastError();
}

}  // namespace lmsae
