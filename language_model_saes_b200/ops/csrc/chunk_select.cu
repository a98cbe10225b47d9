// Batch-level selection of stored pre-activations whose maxima per 32 columns are known (sm_100a).
//
// The encoder GEMM that stores the gated pre-activations of a batch-level top-k leaves the maximum of every 32 columns beside them
// (EncGemmParams::maxima): a sixteenth of the matrix's bytes, and the passes over the matrix (histogram above a floor, counts, lists)
// look at those first and read only the groups that reach the value in question: one in thirty for 64 codes of 65536 columns.
//   4096 x 65536, k 64: histogram 250 -> 98 us, counts and lists 379 -> 158 us
#include "common.cuh"
#include "kernels.h"

namespace lmsae {

namespace {

constexpr int CS_THREADS = 256, CS_U = 4;  // maxima per lane, and groups in flight, at a time

// Calls visit(column, value, in) for the groups of one row, in ascending order, whose maximum is not below t, all lanes of a warp together:
// lane l has column group * 32 + l (in: it exists).
template <typename Fn>
__device__ __forceinline__ void for_groups(const __nv_bfloat16* __restrict__ xr, const float* __restrict__ mr, int N, float t, int g_begin, int g_end, Fn visit) {
  const int lane = threadIdx.x & 31;
  for (int g0 = g_begin; g0 < g_end; g0 += 32 * CS_U) {
    float m[CS_U];
#pragma unroll
    for (int u = 0; u < CS_U; ++u) m[u] = g0 + u * 32 + lane < g_end ? __ldg(mr + g0 + u * 32 + lane) : __int_as_float(0xff800000);
#pragma unroll
    for (int u = 0; u < CS_U; ++u) {
      unsigned todo = __ballot_sync(0xffffffffu, !(m[u] < t) && g0 + u * 32 + lane < g_end);  // (a NaN is looked at)
      while (todo != 0u) {
        int col[CS_U];
        float f[CS_U];
#pragma unroll
        for (int i = 0; i < CS_U; ++i) {
          col[i] = -1;
          f[i] = 0.0f;
          if (todo != 0u) {
            col[i] = (g0 + u * 32 + __ffs(todo) - 1) * 32 + lane;
            todo &= todo - 1u;
            if (col[i] < N) f[i] = __bfloat162float(xr[col[i]]);
          }
        }
#pragma unroll
        for (int i = 0; i < CS_U; ++i)
          if (col[i] >= 0) visit(col[i], f[i], col[i] < N);
      }
    }
  }
}

}  // namespace

// Values of at least *floor (> 0) into bins of the upper 16 bits. A CTA counts the CH_BINS bins from the floor's on in shared memory (sixteen
// octaves), what is beyond goes to memory directly.
constexpr int CH_BINS = 2048;
__global__ void __launch_bounds__(CS_THREADS)
chunk_hist_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ maxima, long long ld_maxima, int B, int N, const float* __restrict__ floor,
                  unsigned* __restrict__ hist, int nbins) {
  pdl_wait();
  __shared__ unsigned s_hist[CH_BINS];
  for (int i = threadIdx.x; i < CH_BINS; i += CS_THREADS) s_hist[i] = 0u;
  __syncthreads();
  const float fl = fmaxf(*floor, 0.0f);
  const uint32_t floor_bits = fl > 0.0f ? __float_as_uint(fl) : 0u, bin0 = floor_bits >> 16;
  const int n_groups = (N + 31) / 32, parts = (n_groups + 32 * CS_U - 1) / (32 * CS_U);
  const long long items = (long long)B * parts, warps = (long long)gridDim.x * (CS_THREADS / 32);
  for (long long it = (long long)blockIdx.x * (CS_THREADS / 32) + (threadIdx.x >> 5); it < items; it += warps) {
    const int row = (int)(it / parts), part = (int)(it - (long long)row * parts);
    for_groups(x + (size_t)row * N, maxima + (size_t)row * ld_maxima, N, fl, part * 32 * CS_U, min(n_groups, (part + 1) * 32 * CS_U),
               [&](int, float f, bool in) {
                 const uint32_t b = in && f > 0.0f ? __float_as_uint(f) : 0u;
                 if (b == 0u || b < floor_bits) return;
                 const uint32_t bin = min(b >> 16, (uint32_t)(nbins - 1));
                 if (bin - bin0 < (uint32_t)CH_BINS) atomicAdd(&s_hist[bin - bin0], 1u);
                 else atomicAdd(hist + bin, 1u);
               });
  }
  __syncthreads();
  for (int i = threadIdx.x; i < CH_BINS; i += CS_THREADS)
    if (s_hist[i] != 0u) atomicAdd(hist + bin0 + i, s_hist[i]);  // (such a bin is below nbins)
}

int chunk_hist_launch(const __nv_bfloat16* x, const float* maxima, long long ld_maxima, int B, int N, const float* floor, unsigned* hist, int nbins,
                      cudaStream_t stream) {
  if (B <= 0 || N <= 0) return 0;
  launch(chunk_hist_kernel, 148 * 8, CS_THREADS, 0, stream, x, maxima, ld_maxima, B, N, floor, hist, nbins);
  return (int)cudaGetLastError();
}

// What row_compact_kernel (select_ops.cu) does with a threshold: per row the number of values above it (a NaN counts as above where the
// threshold is a bf16 value, so that it shows in the loss) and of values equal to it; with `idx`, the lists, equal values up to the row's
// quota. A warp per row.
template <bool LISTS>
__global__ void __launch_bounds__(CS_THREADS)
chunk_compact_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ maxima, long long ld_maxima, int B, int N, const float* __restrict__ thr,
                     const float* __restrict__ col_div, int* __restrict__ nnz, int* __restrict__ ties, const int* __restrict__ tie_quota, int cap,
                     int* __restrict__ idx, float* __restrict__ val) {
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int row = blockIdx.x * (CS_THREADS / 32) + (threadIdx.x >> 5);
  if (row >= B) return;
  const float t = *thr;
  const bool keep_nan = t > 0.0f && __bfloat162float(__float2bfloat16(t)) == t;
  const int quota = LISTS ? tie_quota[row] : 0;
  int n_s = 0, n_t = 0;
  for_groups(x + (size_t)row * N, maxima + (size_t)row * ld_maxima, N, t, 0, (N + 31) / 32, [&](int c, float f, bool in) {
    const bool strict = in && (keep_nan ? !(f <= t) : f > t), tie = in && f == t;
    const unsigned bs = __ballot_sync(0xffffffffu, strict), bt = __ballot_sync(0xffffffffu, tie);
    if constexpr (LISTS) {
      const int tie_rank = n_t + __popc(bt & below);
      const int slot = n_s + __popc(bs & below) + min(tie_rank, quota);
      if ((strict || (tie && tie_rank < quota)) && slot < cap) {
        idx[(size_t)row * cap + slot] = c;
        val[(size_t)row * cap + slot] = col_div != nullptr ? f / col_div[c] : f;
      }
    }
    n_s += __popc(bs);
    n_t += __popc(bt);
  });
  if constexpr (LISTS) {
    const int count = n_s + min(n_t, quota);
    if (lane == 0) nnz[row] = count;
    for (int j = count + lane; j < cap; j += 32) {
      idx[(size_t)row * cap + j] = -1;
      val[(size_t)row * cap + j] = 0.0f;
    }
  } else if (lane == 0) {
    nnz[row] = n_s;
    ties[row] = n_t;
  }
}

int chunk_compact_launch(const __nv_bfloat16* x, const float* maxima, long long ld_maxima, int B, int N, const float* thr, const float* col_div, int* nnz,
                         int* ties, const int* tie_quota, int cap, int* idx, float* val, cudaStream_t stream) {
  if (B <= 0 || N <= 0) return 0;
  const int blocks = (B + CS_THREADS / 32 - 1) / (CS_THREADS / 32);
  if (idx != nullptr) {
    if (tie_quota == nullptr || cap <= 0) return (int)cudaErrorInvalidValue;
    launch(chunk_compact_kernel<true>, blocks, CS_THREADS, 0, stream, x, maxima, ld_maxima, B, N, thr, col_div, nnz, nullptr, tie_quota, cap, idx, val);
  } else {
    if (ties == nullptr) return (int)cudaErrorInvalidValue;
    launch(chunk_compact_kernel<false>, blocks, CS_THREADS, 0, stream, x, maxima, ld_maxima, B, N, thr, nullptr, nnz, ties, nullptr, 0, nullptr, nullptr);
  }
  return (int)cudaGetLastError();
}

}  // namespace lmsae
