// Batch-level selection of stored pre-activations whose maxima per 32 columns are known (sm_100a).
//
// The encoder GEMM that stores the gated pre-activations of a batch-level top-k leaves the maximum of every 32 columns beside them
// (EncGemmParams::maxima): a sixteenth of the matrix's bytes, and the passes over the matrix (histogram above a floor, counts, lists)
// look at those first and read only the groups that reach the value in question: one in thirty for 64 codes of 65536 columns.
// 4096 x 65536, k 64, us; whole matrix, a group at a time with a lane per column and lists in two passes, eight groups at a time and lists in one pass:
//   histogram above the floor 250 -> 98 -> 62 (142 -> 75 in a step), counts and lists 379 -> 158 -> 62
// Bound by the latency of the groups' loads: the bytes (33 MB of maxima, 45 MB of groups at nine tenths of the threshold) take 12 us.
#include <limits.h>
#include "common.cuh"
#include "kernels.h"

namespace lmsae {

namespace {

constexpr int CS_THREADS = 256, CS_U = 4;          // maxima per lane at a time
constexpr int CS_WARPS = CS_THREADS / 32, CS_SPAN = 32 * CS_U;  // groups whose maxima a warp looks at together

// Values [8 * (lane % 4), + 8) of eight groups of 32 columns at a time, a group to four lanes: for the groups [g_begin, g_end) of one row whose
// maximum is not below t, in ascending order, calls visit(column, raw, n) with all lanes of a warp together, where raw holds the bf16 values of
// columns [column, column + n) (n 0 to 8; none: column past the row). The groups of a span are listed first, so that most calls
// find eight of them (a group at a time, a lane per column: 73 instructions a group and a call for 1.1 values above a floor).
template <typename Fn>
__device__ __forceinline__ void for_groups(const __nv_bfloat16* __restrict__ xr, const float* __restrict__ mr, int N, bool vec, float t, int g_begin, int g_end,
                                           unsigned short* list, Fn visit) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  for (int g0 = g_begin; g0 < g_end; g0 += CS_SPAN) {
    float m[CS_U];
#pragma unroll
    for (int u = 0; u < CS_U; ++u) m[u] = g0 + u * 32 + lane < g_end ? __ldg(mr + g0 + u * 32 + lane) : __int_as_float(0xff800000);
    int n = 0;
#pragma unroll
    for (int u = 0; u < CS_U; ++u) {
      const bool in = !(m[u] < t) && g0 + u * 32 + lane < g_end;  // (a NaN is looked at)
      const unsigned mask = __ballot_sync(0xffffffffu, in);
      if (in) list[n + __popc(mask & below)] = (unsigned short)(u * 32 + lane);
      n += __popc(mask);
    }
    __syncwarp();
    for (int i0 = 0; i0 < n; i0 += 16) {  // two calls' values on their way at once
      int col[2], have[2];
      uint4 raw[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = i0 + h * 8 + (lane >> 2);
        col[h] = N;
        have[h] = 0;
        raw[h] = make_uint4(0u, 0u, 0u, 0u);
        if (i < n) {
          col[h] = (g0 + (int)list[i]) * 32 + (lane & 3) * 8;
          have[h] = max(0, min(8, N - col[h]));
          if (vec) {
            if (have[h] > 0) raw[h] = __ldg(reinterpret_cast<const uint4*>(xr + col[h]));
          } else {
            unsigned short v[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] = j < have[h] ? reinterpret_cast<const unsigned short*>(xr)[col[h] + j] : (unsigned short)0;
            raw[h] = make_uint4(v[0] | (uint32_t)v[1] << 16, v[2] | (uint32_t)v[3] << 16, v[4] | (uint32_t)v[5] << 16, v[6] | (uint32_t)v[7] << 16);
          }
        }
      }
      visit(col[0], raw[0], have[0]);
      if (i0 + 8 < n) visit(col[1], raw[1], have[1]);
    }
    __syncwarp();  // (the list is written again)
  }
}
__device__ __forceinline__ unsigned raw_value(const uint4& r, int j) {
  const uint32_t w = j < 2 ? r.x : j < 4 ? r.y : j < 6 ? r.z : r.w;
  return j & 1 ? w >> 16 : w & 0xffffu;
}

}  // namespace

// Values of at least *floor (> 0) into bins of the upper 16 bits. A CTA counts the CH_BINS bins from the floor's on in shared memory (sixteen
// octaves), what is beyond goes to memory directly.
constexpr int CH_BINS = 2048;
__global__ void __launch_bounds__(CS_THREADS)
chunk_hist_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ maxima, long long ld_maxima, int B, int N, const float* __restrict__ floor,
                  unsigned* __restrict__ hist, int nbins, bool vec) {
  pdl_wait();
  __shared__ unsigned s_hist[CH_BINS];
  __shared__ unsigned short s_list[CS_WARPS][CS_SPAN];
  for (int i = threadIdx.x; i < CH_BINS; i += CS_THREADS) s_hist[i] = 0u;
  __syncthreads();
  const float fl = fmaxf(*floor, 0.0f);
  const uint32_t floor_bits = fl > 0.0f ? __float_as_uint(fl) : 0u, bin0 = floor_bits >> 16;
  // a bf16 value counts from the first that is not below the floor (and positive) up to infinity
  const uint32_t first = max((floor_bits + 0xffffu) >> 16, 1u), most = 0x7f80u;
  const int n_groups = (N + 31) / 32, parts = (n_groups + CS_SPAN - 1) / CS_SPAN;
  const long long items = (long long)B * parts, warps = (long long)gridDim.x * CS_WARPS;
  for (long long it = (long long)blockIdx.x * CS_WARPS + (threadIdx.x >> 5); it < items; it += warps) {
    const int row = (int)(it / parts), part = (int)(it - (long long)row * parts);
    for_groups(x + (size_t)row * N, maxima + (size_t)row * ld_maxima, N, vec, fl, part * CS_SPAN, min(n_groups, (part + 1) * CS_SPAN),
               s_list[threadIdx.x >> 5], [&](int, const uint4& raw, int n) {
                 unsigned in = 0u;
#pragma unroll
                 for (int j = 0; j < 8; ++j) in |= (j < n && raw_value(raw, j) >= first && raw_value(raw, j) <= most) ? 1u << j : 0u;
                 while (in != 0u) {
                   const int j = __ffs(in) - 1;
                   in &= in - 1u;
                   const uint32_t bin = min(raw_value(raw, j), (uint32_t)(nbins - 1));
                   if (bin - bin0 < (uint32_t)CH_BINS) atomicAdd(&s_hist[bin - bin0], 1u);
                   else atomicAdd(hist + bin, 1u);
                 }
               });
  }
  __syncthreads();
  for (int i = threadIdx.x; i < CH_BINS; i += CS_THREADS)
    if (s_hist[i] != 0u) atomicAdd(hist + bin0 + i, s_hist[i]);  // (such a bin is below nbins)
}

static bool rows_aligned(const __nv_bfloat16* x, int N) { return N % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0; }

int chunk_hist_launch(const __nv_bfloat16* x, const float* maxima, long long ld_maxima, int B, int N, const float* floor, unsigned* hist, int nbins,
                      cudaStream_t stream) {
  if (B <= 0 || N <= 0) return 0;
  launch(chunk_hist_kernel, 148 * 8, CS_THREADS, 0, stream, x, maxima, ld_maxima, B, N, floor, hist, nbins, rows_aligned(x, N));
  return (int)cudaGetLastError();
}

// What row_compact_kernel (select_ops.cu) does with a threshold: per row the number of values above it (a NaN counts as above where the
// threshold is a bf16 value, so that it shows in the loss) and of values equal to it; with lists, those values in ascending order of
// columns, equal ones up to the row's quota. A warp per row.
struct RowList {
  int* idx;
  float* val;
  int cap;
};
template <bool LISTS>
__device__ __forceinline__ void compact_row(const __nv_bfloat16* __restrict__ xr, const float* __restrict__ mr, int N, bool vec, float t, const float* __restrict__ col_div,
                                            int quota, const RowList& to, unsigned short* list, int& n_s, int& n_t) {
  const int lane = threadIdx.x & 31;
  const bool keep_nan = t > 0.0f && __bfloat162float(__float2bfloat16(t)) == t;
  n_s = n_t = 0;
  for_groups(xr, mr, N, vec, t, 0, (N + 31) / 32, list, [&](int c, const uint4& raw, int n) {
    unsigned strict = 0u, tie = 0u;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float f = __uint_as_float(raw_value(raw, j) << 16);
      strict |= (j < n && (keep_nan ? !(f <= t) : f > t)) ? 1u << j : 0u;
      tie |= (j < n && f == t) ? 1u << j : 0u;
    }
    // counts of the lanes before this one: strict ones in the lower half, equal ones in the upper (at most 256 each)
    const unsigned mine = (unsigned)__popc(strict) | (unsigned)__popc(tie) << 16;
    if constexpr (LISTS) {
      unsigned sum = mine;
#pragma unroll
      for (int o = 1; o < 32; o *= 2) {
        const unsigned v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
      }
      const unsigned before = sum - mine;
      int s = n_s + (int)(before & 0xffffu), e = n_t + (int)(before >> 16);
      for (unsigned in = strict | tie; in != 0u; in &= in - 1u) {
        const int j = __ffs(in) - 1;
        const bool equal = (tie >> j & 1u) != 0u;
        const int slot = s + min(e, quota);
        if ((!equal || e < quota) && slot < to.cap) {
          const float f = __uint_as_float(raw_value(raw, j) << 16);
          to.idx[slot] = c + j;
          to.val[slot] = col_div != nullptr ? f / col_div[c + j] : f;
        }
        if (equal) ++e;
        else ++s;
      }
      const unsigned total = __shfl_sync(0xffffffffu, sum, 31);
      n_s += (int)(total & 0xffffu);
      n_t += (int)(total >> 16);
    } else {
      const unsigned total = __reduce_add_sync(0xffffffffu, mine);
      n_s += (int)(total & 0xffffu);
      n_t += (int)(total >> 16);
    }
  });
}
__device__ __forceinline__ void pad_row(const RowList& to, int count) {
  for (int j = count + (int)(threadIdx.x & 31); j < to.cap; j += 32) {
    to.idx[j] = -1;
    to.val[j] = 0.0f;
  }
}

template <bool LISTS>
__global__ void __launch_bounds__(CS_THREADS)
chunk_compact_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ maxima, long long ld_maxima, int B, int N, bool vec, const float* __restrict__ thr,
                     const float* __restrict__ col_div, int* __restrict__ nnz, int* __restrict__ ties, const int* __restrict__ tie_quota, int cap,
                     int* __restrict__ idx, float* __restrict__ val) {
  pdl_wait();
  __shared__ unsigned short s_list[CS_WARPS][CS_SPAN];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = blockIdx.x * CS_WARPS + warp;
  if (row >= B) return;
  // (lists without quotas: all equal values, whose number is wanted too)
  const int quota = LISTS ? tie_quota != nullptr ? tie_quota[row] : INT_MAX : 0;
  const RowList to = {LISTS ? idx + (size_t)row * cap : nullptr, LISTS ? val + (size_t)row * cap : nullptr, cap};
  int n_s, n_t;
  compact_row<LISTS>(x + (size_t)row * N, maxima + (size_t)row * ld_maxima, N, vec, *thr, col_div, quota, to, s_list[warp], n_s, n_t);
  if constexpr (LISTS) {
    const int count = n_s + min(n_t, quota);
    pad_row(to, count);
    if (lane == 0) nnz[row] = tie_quota != nullptr ? count : n_s;
    if (lane == 0 && ties != nullptr) ties[row] = n_t;
  } else if (lane == 0) {
    nnz[row] = n_s;
    ties[row] = n_t;
  }
}

// Places for equal values, n_ties of them for all rows, in the order of the rows: quota[row]. One CTA. (Sums in 64 bits: rows of 2^19 equal
// values reach 2^31 within a turn of 4096.)
__global__ void __launch_bounds__(1024)
tie_quota_kernel(const int* __restrict__ ties, const long long* __restrict__ n_ties, int B, int* __restrict__ quota) {
  pdl_wait();
  __shared__ long long s_sum[32];
  __shared__ long long s_total;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  long long left = *n_ties;
  for (int r0 = 0; r0 < B; r0 += 4096) {
    int t[4];
    long long mine = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + (int)threadIdx.x * 4 + i;
      t[i] = r < B ? ties[r] : 0;
      mine += t[i];
    }
    long long sum = mine;
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      const long long v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    if (lane == 31) s_sum[warp] = sum;
    __syncthreads();
    if (warp == 0) {
      long long w = s_sum[lane];
#pragma unroll
      for (int o = 1; o < 32; o *= 2) {
        const long long v = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += v;
      }
      s_sum[lane] = w;
      if (lane == 31) s_total = w;
    }
    __syncthreads();
    long long before = sum - mine + (warp > 0 ? s_sum[warp - 1] : 0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + (int)threadIdx.x * 4 + i;
      if (r < B) quota[r] = (int)min((long long)t[i], max(0LL, left - before));
      before += t[i];
    }
    left -= s_total;
    __syncthreads();
  }
}

// Takes the equal values beyond a row's quota out of lists that hold them all (a row whose list they overflowed is made again), and leaves the rows'
// counts; rows with more than cap are counted in overflow. A warp per row, and little to do: most rows have all or none of a few such values.
__global__ void __launch_bounds__(CS_THREADS)
trim_ties_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ maxima, long long ld_maxima, int B, int N, bool vec, const float* __restrict__ thr,
                 const float* __restrict__ col_div, int* __restrict__ nnz, const int* __restrict__ ties, const int* __restrict__ tie_quota, int cap,
                 int* __restrict__ idx, float* __restrict__ val, unsigned long long* __restrict__ overflow) {
  pdl_wait();
  __shared__ unsigned short s_list[CS_WARPS][CS_SPAN];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = blockIdx.x * CS_WARPS + warp;
  if (row >= B) return;
  const int n_s = nnz[row], n_t = ties[row], quota = tie_quota[row], count = n_s + quota;
  const RowList to = {idx + (size_t)row * cap, val + (size_t)row * cap, cap};
  const __nv_bfloat16* xr = x + (size_t)row * N;
  if (quota < n_t) {
    if (n_s + n_t > cap) {
      int s, e;
      compact_row<true>(xr, maxima + (size_t)row * ld_maxima, N, vec, *thr, col_div, quota, to, s_list[warp], s, e);
    } else {
      const float t = *thr;
      int kept = 0, equal = 0;
      for (int base = 0; base < n_s + n_t; base += 32) {
        const bool in = base + lane < n_s + n_t;
        const int c = in ? to.idx[base + lane] : 0;
        const float v = in ? to.val[base + lane] : 0.0f;
        const bool tie = in && __bfloat162float(xr[c]) == t;
        const unsigned bt = __ballot_sync(0xffffffffu, tie), below = (1u << lane) - 1u;
        const bool keep = in && (!tie || equal + __popc(bt & below) < quota);
        const unsigned bk = __ballot_sync(0xffffffffu, keep);
        __syncwarp();  // (read before anything at or behind it is overwritten)
        if (keep) {
          const int slot = kept + __popc(bk & below);
          to.idx[slot] = c;
          to.val[slot] = v;
        }
        kept += __popc(bk);
        equal += __popc(bt);
      }
    }
    __syncwarp();
    pad_row(to, count);
  }
  if (lane == 0) {
    nnz[row] = count;
    if (overflow != nullptr && count > cap) atomicAdd(overflow, 1ULL);
  }
}

int chunk_compact_launch(const __nv_bfloat16* x, const float* maxima, long long ld_maxima, int B, int N, const float* thr, const float* col_div, int* nnz,
                         int* ties, const int* tie_quota, int cap, int* idx, float* val, cudaStream_t stream) {
  if (B <= 0 || N <= 0) return 0;
  const int blocks = (B + CS_WARPS - 1) / CS_WARPS;
  const bool vec = rows_aligned(x, N);
  if (idx != nullptr) {
    if (tie_quota == nullptr || cap <= 0) return (int)cudaErrorInvalidValue;
    launch(chunk_compact_kernel<true>, blocks, CS_THREADS, 0, stream, x, maxima, ld_maxima, B, N, vec, thr, col_div, nnz, nullptr, tie_quota, cap, idx, val);
  } else {
    if (ties == nullptr) return (int)cudaErrorInvalidValue;
    launch(chunk_compact_kernel<false>, blocks, CS_THREADS, 0, stream, x, maxima, ld_maxima, B, N, vec, thr, nullptr, nnz, ties, nullptr, 0, nullptr, nullptr);
  }
  return (int)cudaGetLastError();
}

// Counts, quotas and lists with one pass over the matrix: the lists with all equal values, then the quotas, then what is beyond them is taken out.
// ties, quota: scratch [B]
int chunk_lists_launch(const __nv_bfloat16* x, const float* maxima, long long ld_maxima, int B, int N, const float* thr, const long long* n_ties,
                       const float* col_div, int* nnz, int* ties, int* quota, int cap, int* idx, float* val, unsigned long long* overflow, cudaStream_t stream) {
  if (B <= 0 || N <= 0) return 0;
  if (cap <= 0) return (int)cudaErrorInvalidValue;
  const int blocks = (B + CS_WARPS - 1) / CS_WARPS;
  const bool vec = rows_aligned(x, N);
  launch(chunk_compact_kernel<true>, blocks, CS_THREADS, 0, stream, x, maxima, ld_maxima, B, N, vec, thr, col_div, nnz, ties, nullptr, cap, idx, val);
  launch(tie_quota_kernel, 1, 1024, 0, stream, ties, n_ties, B, quota);
  launch(trim_ties_kernel, blocks, CS_THREADS, 0, stream, x, maxima, ld_maxima, B, N, vec, thr, col_div, nnz, ties, quota, cap, idx, val, overflow);
  return (int)cudaGetLastError();
}

// JumpReLU: the values above their column's threshold, in ascending order of columns, up to cap of them; rows with more are counted in overflow. The maxima
// are those of the values times a gate (jumprelu_begin_kernel): a group that holds such a value reaches 1 less two roundings, and every value is compared
// with its threshold. A warp per row; what is left of a row is the latency of its spans of maxima. 64 codes a row, whole matrix -> by maxima: 4096 x 18432
// 51 -> 20 us, 4096 x 98304 228 -> 69.
__global__ void __launch_bounds__(CS_THREADS)
chunk_columns_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ maxima, long long ld_maxima, int B, int N, const float* __restrict__ col_thr, int cap,
                     int* __restrict__ idx, float* __restrict__ val, unsigned long long* __restrict__ overflow) {
  pdl_wait();
  __shared__ unsigned short s_list[CS_WARPS][CS_SPAN];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row = blockIdx.x * CS_WARPS + warp;
  if (row >= B) return;
  const RowList to = {idx + (size_t)row * cap, val + (size_t)row * cap, cap};
  int n = 0;
  auto visit = [&](int c, const uint4& raw, int have) {
    float t[8];
    if (have > 0) {  // (eight columns: N % 8 == 0)
      const float4 a = __ldg(reinterpret_cast<const float4*>(col_thr + c)), b = __ldg(reinterpret_cast<const float4*>(col_thr + c) + 1);
      t[0] = a.x; t[1] = a.y; t[2] = a.z; t[3] = a.w; t[4] = b.x; t[5] = b.y; t[6] = b.z; t[7] = b.w;
    }
    unsigned in = 0u;
#pragma unroll
    for (int j = 0; j < 8; ++j) in |= (have > 0 && __uint_as_float(raw_value(raw, j) << 16) > t[j]) ? 1u << j : 0u;
    int sum = __popc(in);
#pragma unroll
    for (int o = 1; o < 32; o *= 2) {
      const int v = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += v;
    }
    int slot = n + sum - __popc(in);
    n += __shfl_sync(0xffffffffu, sum, 31);
    for (; in != 0u; in &= in - 1u, ++slot) {
      const int j = __ffs(in) - 1;
      if (slot < cap) {
        to.idx[slot] = c + j;
        to.val[slot] = __uint_as_float(raw_value(raw, j) << 16);
      }
    }
  };
  // (a row with more values than places is looked at up to where that shows)
  const int groups = (N + 31) / 32;
  for (int g0 = 0; g0 < groups && n <= cap; g0 += CS_SPAN)
    for_groups(x + (size_t)row * N, maxima + (size_t)row * ld_maxima, N, true, 0.9999f, g0, min(groups, g0 + CS_SPAN), s_list[warp], visit);
  pad_row(to, n);
  if (lane == 0 && n > cap) atomicAdd(overflow, 1ULL);
}

int chunk_columns_launch(const __nv_bfloat16* x, const float* maxima, long long ld_maxima, int B, int N, const float* col_thr, int cap, int* idx, float* val,
                         unsigned long long* overflow, cudaStream_t stream) {
  if (B <= 0 || N <= 0 || cap <= 0 || !rows_aligned(x, N) || reinterpret_cast<uintptr_t>(col_thr) % 16 != 0) return (int)cudaErrorInvalidValue;
  return (int)launch(chunk_columns_kernel, (B + CS_WARPS - 1) / CS_WARPS, CS_THREADS, 0, stream, x, maxima, ld_maxima, B, N, col_thr, cap, idx, val, overflow);
}

}  // namespace lmsae
