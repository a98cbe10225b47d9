// Exact top-k merge of per-range candidate lists.
//
// The encoder GEMM emits, for every row, C = (number of ranges) * KS candidates (gated value, column or
// -1). This kernel keeps the k best (value descending, ties by position). Under feature
// sharding it runs twice: once per rank on its own ranges (emit_gated = 1, output = k (g, local column)
// pairs that are exchanged between the shards), and once on the gathered lists of all shards, where only
// candidates in [own_lo, own_hi) -- this shard's segment -- are written out; positions won by other
// shards stay (-1, 0). That reproduces a global per-row TopK over the sharded feature axis (the job of
// distributed_topk in utils/distributed/ops.py:158-266 of the reference) with one exchange instead of
// an iterative threshold search.
#include "comm_common.cuh"
#include "fp32_exact.cuh"

namespace lmsae {

constexpr int MERGE_WARPS = 4;  // (fewer where their candidates do not fit)

// One warp per row. Positive floats order like their bit patterns, so the k-th largest candidate is found by a
// descent over the 31 value bits instead of ranking every candidate against every other one: two bits per step, the three counts of a
// step in one word and one warp reduction, until exactly k are left; candidates equal to the threshold get the remaining places in slot
// order. The (at most k) winners are compacted into shared memory in slot order and ranked among themselves. Only winners whose
// candidate slot lies in [own_lo, own_hi) are written, in value-descending order FROM SLOT 0 ON (the rest of the row is
// (-1, 0)): consumers of a shard's codes may stop at the first empty slot.
// All rows are in flight at once: what bounds it is the latency of a warp's chain. PER candidates per lane are held in registers (up to 768 of
// them; more, as small batches with many ranges have, come from shared memory and take a step per bit). 4096 rows of 256 candidates, k
// 50: 25 us with candidates in shared memory, a step per bit and slots compared in the ranking -> 14 us; 512 of 32, k 8: 9.6 -> 4.1.
//
// comm.mode selects what surrounds the merge under feature sharding:
//   kMergeLocal  nothing (single GPU, or lists that are exchanged by other means)
//   kMergePush   the row's k (value, column) pairs are not written to out_* but stored straight into segment
//                [rank * k, (rank + 1) * k) of EVERY rank's merge input (the all-gather of the candidate lists by
//                peer stores, fused into the kernel that produces them); the last block publishes the epoch
//   kMergeWait   the kernel first waits (bounded) until every rank has published the epoch for the candidate
//                phase, then merges the gathered lists it finds in this rank's own buffer
template <int PER>
__global__ void __launch_bounds__(MERGE_WARPS * 32)
topk_merge_kernel(const float* cand_val, const int* cand_idx, int M, int C, int k,  // may be peer-written: no read-only path
                  const float* __restrict__ gate, int own_lo, int own_hi, int emit_gated,
                  int* __restrict__ out_idx, float* __restrict__ out_val, const MergeComm comm) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  // per warp: winner keys[k] and ids[k], staged output ids[k] and values[k], and where candidates are not in registers keys[C], ids[C]
  uint32_t* wkey = reinterpret_cast<uint32_t*>(smem_raw) + (size_t)warp * (4 * k + (PER == 0 ? 2 * C : 0));
  int* wid = reinterpret_cast<int*>(wkey + k);
  int* oidx = wid + k;
  float* oval = reinterpret_cast<float*>(oidx + k);
  uint32_t* skey = reinterpret_cast<uint32_t*>(oval + k);
  int* sidx = reinterpret_cast<int*>(skey + C);

  bool inputs_ok = true;
  if (comm.mode == kMergeWait) inputs_ok = wait_all_sources(comm.pt, kPhaseCand, comm.epoch, comm.status);

  const int warps = blockDim.x >> 5;
  for (int row = blockIdx.x * warps + warp; row < M; row += gridDim.x * warps) {
    int n_own = 0;
    if (inputs_ok) {
      const float* cv = cand_val + (size_t)row * C;
      const int* ci = cand_idx + (size_t)row * C;
      uint32_t key[PER > 0 ? PER : 1];
      int id[PER > 0 ? PER : 1];
      if constexpr (PER > 0) {
#pragma unroll
        for (int i = 0; i < PER; ++i) {
          const int c = i * 32 + lane;
          id[i] = c < C ? ci[c] : -1;
          key[i] = c < C ? __float_as_uint(cv[c]) : 0u;
        }
#pragma unroll
        for (int i = 0; i < PER; ++i) key[i] = (id[i] >= 0 && __uint_as_float(key[i]) > 0.0f) ? key[i] : 0u;  // only positive candidates compete
      } else {
        for (int i = lane; i < C; i += 32) {
          const int d = ci[i];
          const float v = cv[i];
          sidx[i] = d;
          skey[i] = (d >= 0 && v > 0.0f) ? __float_as_uint(v) : 0u;
        }
        __syncwarp();
      }
      // threshold: the largest t with count(key >= t) >= k (0 when fewer than k candidates are positive), or one that exactly k reach
      uint32_t t = 0;
      bool exactly = false;
      int above = 0;
      if constexpr (PER > 0) {
        for (int shift = 30; shift >= 0 && !exactly; shift -= 2) {  // (bit 31 is never set)
          const uint32_t t1 = t | (1u << shift), t2 = t | (2u << shift), t3 = t | (3u << shift);
          unsigned n = 0;
#pragma unroll
          for (int i = 0; i < PER; ++i) n += (unsigned)(key[i] >= t1) + ((unsigned)(key[i] >= t2) << 10) + ((unsigned)(key[i] >= t3) << 20);
          n = __reduce_add_sync(0xffffffffu, n);
          const int c1 = (int)(n & 1023u), c2 = (int)((n >> 10) & 1023u), c3 = (int)(n >> 20);
          if (c3 >= k) { t = t3; exactly = c3 == k; }
          else if (c2 >= k) { t = t2; exactly = c2 == k; }
          else if (c1 >= k) { t = t1; exactly = c1 == k; }
        }
        if (!exactly && t != 0u) {
#pragma unroll
          for (int i = 0; i < PER; ++i) above += key[i] > t;
        }
      } else {
        for (int bit = 30; bit >= 0; --bit) {
          const uint32_t trial = t | (1u << bit);
          int c = 0;
          for (int i = lane; i < C; i += 32) c += skey[i] >= trial;
          if (__reduce_add_sync(0xffffffffu, c) >= k) t = trial;
        }
        for (int i = lane; i < C; i += 32) above += skey[i] > t;
      }
      const int ties_wanted = exactly ? k : t == 0u ? 0 : k - __reduce_add_sync(0xffffffffu, above);  // (t == 0: nothing equals t)
      // compaction of the winners in slot order; [own0, own1) of them lie in this shard's slots
      int n_win = 0, ties_seen = 0, own0 = 0, own1 = 0;
      auto take = [&](int base, uint32_t u, int d) {
        const bool eq = t != 0u && u == t;
        const unsigned eq_ballot = __ballot_sync(0xffffffffu, eq);
        const bool win = u > t || (eq && ties_seen + __popc(eq_ballot & lt_mask) < ties_wanted);
        const unsigned win_ballot = __ballot_sync(0xffffffffu, win);
        if (win) {
          const int pos = n_win + __popc(win_ballot & lt_mask);
          wkey[pos] = u;
          wid[pos] = d;
        }
        const int slot = base + lane;
        own0 += __popc(__ballot_sync(0xffffffffu, win && slot < own_lo));
        own1 += __popc(__ballot_sync(0xffffffffu, win && slot < own_hi));
        n_win += __popc(win_ballot);
        ties_seen += __popc(eq_ballot);
      };
      if constexpr (PER > 0) {
#pragma unroll
        for (int i = 0; i < PER; ++i) take(i * 32, key[i], id[i]);
      } else {
        for (int base = 0; base < C; base += 32) take(base, base + lane < C ? skey[base + lane] : 0u, base + lane < C ? sidx[base + lane] : -1);
      }
      __syncwarp();
      // place of each of this shard's winners among this shard's winners (value descending, earlier slot first among equals)
      n_own = own1 - own0;
      for (int w = own0 + lane; w < own1; w += 32) {
        const uint32_t u = wkey[w];
        const int d = wid[w];
        int place = 0;
#pragma unroll 8
        for (int j = own0; j < own1; ++j) place += wkey[j] + (j < w ? 1u : 0u) > u;  // (a key's successor is no overflow: keys are below 2^31)
        const float v = __uint_as_float(u);
        oidx[place] = d;
        oval[place] = (!emit_gated && gate != nullptr) ? v / gate[d] : v;
      }
    }
    for (int i = n_own + lane; i < k; i += 32) {
      oidx[i] = -1;
      oval[i] = 0.0f;
    }
    __syncwarp();
    if (comm.mode == kMergePush) {
      const size_t o = (size_t)row * ((size_t)comm.pt.world * k) + (size_t)comm.pt.rank * k;
      for (int p = 0; p < comm.pt.world; ++p) {
        float* dv = reinterpret_cast<float*>(comm.pt.base[p] + comm.pt.cand_val_off) + o;
        int* di = reinterpret_cast<int*>(comm.pt.base[p] + comm.pt.cand_idx_off) + o;
        for (int i = lane; i < k; i += 32) {
          dv[i] = oval[i];
          di[i] = oidx[i];
        }
      }
    } else {
      for (int i = lane; i < k; i += 32) {
        out_idx[(size_t)row * k + i] = oidx[i];
        out_val[(size_t)row * k + i] = oval[i];
      }
    }
    __syncwarp();
  }
  if (comm.mode == kMergePush) signal_peers_when_grid_done(comm.pt, kPhaseCand, comm.epoch, comm.done_counter);
}

int topk_merge_launch(const float* cand_val, const int* cand_idx, int M, int C, int k, const float* gate,
                      int own_lo, int own_hi, int emit_gated, int* out_idx, float* out_val, const MergeComm& comm,
                      cudaStream_t stream) {
  const int per = C <= 128 ? 4 : C <= 256 ? 8 : C <= 512 ? 16 : C <= 768 ? 24 : 0;
  // Up to 128 rows have 148 ranges, and 64 candidates of each are 74 KB a row: two rows a CTA.
  const size_t warp_bytes = (4 * (size_t)k + (per == 0 ? 2 * (size_t)C : 0)) * 4;
  int warps = MERGE_WARPS;
  while (warps > 1 && warps * warp_bytes > 200 * 1024) warps /= 2;
  const size_t smem = warps * warp_bytes;
  if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;
  if (comm.mode != kMergePush && (out_idx == nullptr || out_val == nullptr)) return (int)cudaErrorInvalidValue;
  auto kern = per == 4 ? topk_merge_kernel<4> : per == 8 ? topk_merge_kernel<8> : per == 16 ? topk_merge_kernel<16> : per == 24 ? topk_merge_kernel<24> : topk_merge_kernel<0>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  int blocks = (M + warps - 1) / warps;
  if (blocks > 148 * 8) blocks = 148 * 8;
  launch(kern, blocks, warps * 32, smem, stream, cand_val, cand_idx, M, C, k, gate, own_lo, own_hi,
                                                  emit_gated, out_idx, out_val, comm);
  return (int)cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------
// Row top-k over a materialised bf16 matrix H[M, N] (used when k is larger than the fused epilogue
// supports, for Aux-K over dead features and for the generic autograd path).
// value = H * gate (gate optional) * alive (alive optional byte mask: only features with alive != 0
// compete); only values > 0 compete.
//
// One CTA per row, bound by reading the row (twice, the second time from L1 / L2). Pass 1 keeps the maxima of 2048 disjoint
// groups of columns in registers; at least k values of the row are at or above the k-th largest of them (16 leading bits
// of it are enough), and for k well below 2048 hardly more than k are. Pass 2 collects the columns at or above that bound in
// shared memory, where the exact k-th value is found by a descent over the value bits. Rows whose bound lets too many through
// (values repeated thousands of times) and k > 1024 take a radix descent over the row itself: four histogram passes.
// 4096 rows of 32768 gated columns, k 128: 546 us (histograms for every row) -> 196 us; 2048 x 8192: 125 -> 58 us.
// ------------------------------------------------------------------------------------------------
constexpr int RT_THREADS = 256;  // (what is left of a row's time is latency: five CTAs of 256 threads per SM hide it as well as three of 512 with wider barriers)
constexpr int RT_MAXIMA = 8;     // column groups per thread
constexpr int RT_CAP = 10 * RT_THREADS;  // candidates in shared memory
constexpr int RT_MAX_GROUPS = 1024;  // of 32 columns that reach the bound, where their maxima are known (half as many codes are allowed for)
constexpr int RT_BOUND_K = RT_THREADS * RT_MAXIMA / 2;  // (about 1.4 k candidates there, k + a few for small k)

__device__ __forceinline__ float stored_value(const __nv_bfloat16* p) { return __bfloat162float(*p); }
__device__ __forceinline__ float stored_value(const float* p) { return *p; }
template <typename T>
__device__ __forceinline__ float gated_value(const T* __restrict__ hrow, const float* __restrict__ gate,
                                             const uint8_t* __restrict__ alive, int c) {
  float v = stored_value(hrow + c);
  if (gate != nullptr) v *= gate[c];
  if (alive != nullptr && alive[c] == 0) v = 0.0f;
  return v;
}

// the gated values of columns [c, c + 8), zero past the end of the row
__device__ __forceinline__ void gated_values8(const __nv_bfloat16* __restrict__ hrow, const float* __restrict__ gate,
                                              const uint8_t* __restrict__ alive, int c, int N, bool vec, float (&v)[8]) {
  if (vec) {
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(hrow + c));
    const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[2 * i] = __uint_as_float(w[i] << 16);
      v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
    if (gate != nullptr) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(gate + c)), b = __ldg(reinterpret_cast<const float4*>(gate + c) + 1);
      v[0] *= a.x; v[1] *= a.y; v[2] *= a.z; v[3] *= a.w;
      v[4] *= b.x; v[5] *= b.y; v[6] *= b.z; v[7] *= b.w;
    }
    if (alive != nullptr) {
      const uint2 m = __ldg(reinterpret_cast<const uint2*>(alive + c));
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if ((((i < 4 ? m.x : m.y) >> (8 * (i & 3))) & 0xffu) == 0u) v[i] = 0.0f;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = c + i < N ? gated_value(hrow, gate, alive, c + i) : 0.0f;
  }
}

// The radix descent over the row: 4 passes of 8 bits, 256-bin histogram in shared memory, then one pass over the survivors.
template <typename T>
__device__ __noinline__ void row_topk_radix(const T* __restrict__ hrow, int row, int N, int k, const float* __restrict__ gate,
                                            const uint8_t* __restrict__ alive, int* __restrict__ out_idx, float* __restrict__ out_val,
                                            __nv_bfloat16* __restrict__ dense_row = nullptr) {
  __shared__ unsigned hist[256];
  __shared__ unsigned s_prefix, s_remaining, s_count_gt, s_cursor_gt, s_cursor_eq;
  unsigned prefix = 0;     // bits decided so far (from the top)
  unsigned remaining = k;  // how many of the top-k are still inside the undecided bucket
  bool fewer_than_k = false;
  for (int pass = 0; pass < 4; ++pass) {
    const int shift = 24 - 8 * pass;
    for (int i = threadIdx.x; i < 256; i += RT_THREADS) hist[i] = 0;
    __syncthreads();
    const unsigned hi_mask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
    for (int c = threadIdx.x; c < N; c += RT_THREADS) {
      const float v = gated_value(hrow, gate, alive, c);
      if (v > 0.0f) {
        const unsigned b = __float_as_uint(v);
        if ((b & hi_mask) == prefix) atomicAdd(&hist[(b >> shift) & 0xff], 1u);
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned acc = 0;
      int bin = 255;
      for (; bin >= 0; --bin) {
        if (acc + hist[bin] >= remaining) break;
        acc += hist[bin];
      }
      if (bin < 0) {  // fewer than `remaining` positive values in this bucket: keep them all
        s_prefix = 0xffffffffu;
        s_remaining = 0;
      } else {
        s_prefix = prefix | ((unsigned)bin << shift);
        s_remaining = remaining - acc;
      }
    }
    __syncthreads();
    if (s_prefix == 0xffffffffu) {
      fewer_than_k = true;
      break;
    }
    prefix = s_prefix;
    remaining = s_remaining;
    __syncthreads();
  }
  // threshold bit pattern = prefix (exact k-th value); `remaining` = how many equal to it to keep
  const unsigned thr = fewer_than_k ? 0u : prefix;
  if (threadIdx.x == 0) {
    s_cursor_gt = 0;
    s_cursor_eq = 0;
    s_count_gt = fewer_than_k ? 0u : (unsigned)k - remaining;
  }
  for (int i = threadIdx.x; i < k && dense_row == nullptr; i += RT_THREADS) {
    out_idx[(size_t)row * k + i] = -1;
    out_val[(size_t)row * k + i] = 0.0f;
  }
  __syncthreads();
  for (int c = threadIdx.x; c < N; c += RT_THREADS) {
    const float v = gated_value(hrow, gate, alive, c);
    if (v > 0.0f) {
      const unsigned b = __float_as_uint(v);
      int pos = -1;
      if (fewer_than_k || b > thr) {
        pos = (int)atomicAdd(&s_cursor_gt, 1u);
      } else if (b == thr) {
        const unsigned e = atomicAdd(&s_cursor_eq, 1u);
        if (e < remaining) pos = (int)(s_count_gt + e);
      }
      if (pos >= 0 && pos < k) {
        const float a = (gate != nullptr) ? v / gate[c] : v;
        if (dense_row != nullptr) {
          dense_row[c] = __float2bfloat16(a);
        } else {
          out_idx[(size_t)row * k + pos] = c;
          out_val[(size_t)row * k + pos] = a;
        }
      }
    }
  }
}

// The largest t whose lowest `skip` bits are zero with  count(values >= t) >= k  over the CTA (the values' bit patterns are those
// of non-negative floats; fewer than k of them at all: 0). Two bits per step and one barrier: a warp's three counts travel in one
// word, which every warp adds up for itself (atomic sums cost 1500 cycles a step: 217 and 70 us; the words of two steps alternate). Every
// thread returns the same.
constexpr int RT_WARPS = RT_THREADS / 32;
template <int N>
__device__ __forceinline__ unsigned descend(const unsigned (&val)[N], int k, int skip, unsigned (&counts)[2][RT_WARPS]) {
  static_assert(N * 32 < 1024 && RT_WARPS <= 32, "a warp's counts are packed in ten bits each");
  const int lane = threadIdx.x & 31;
  unsigned t = 0;
  __syncthreads();  // (the words may still be read by an earlier call)
  for (int shift = 30; shift >= skip; shift -= 2) {  // (bit 31 is never set)
    const unsigned t1 = t | (1u << shift), t2 = t | (2u << shift), t3 = t | (3u << shift);
    unsigned n = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) n += (unsigned)(val[i] >= t1) + ((unsigned)(val[i] >= t2) << 10) + ((unsigned)(val[i] >= t3) << 20);
    n = __reduce_add_sync(0xffffffffu, n);
    unsigned* words = counts[(shift >> 1) & 1];
    if (lane == 0) words[threadIdx.x >> 5] = n;
    __syncthreads();
    n = lane < RT_WARPS ? words[lane] : 0u;
    const int c1 = (int)__reduce_add_sync(0xffffffffu, n & 1023u), c2 = (int)__reduce_add_sync(0xffffffffu, (n >> 10) & 1023u),
              c3 = (int)__reduce_add_sync(0xffffffffu, n >> 20);
    const int at = c3 >= k ? c3 : c2 >= k ? c2 : c1;
    if (c3 >= k) t = t3;
    else if (c2 >= k) t = t2;
    else if (c1 >= k) t = t1;
    if (at == k) break;
  }
  return t;
}

// MAXIMA: the largest gated value of every 32 columns comes with H (the encoder GEMM's epilogue leaves them): those are the column groups,
// and only groups whose maximum reaches the bound are read at all: 4096 rows of 32768, k 128, with a gate: 195 -> 111 us (211 -> 135 without).
// DENSE: instead of lists the row itself, bf16, zero where nothing was selected (an operand of products over the columns: Aux-K's codes over a dictionary of
// dead features, 4096 rows of 9216, k 512: 136 us and 92 for fill, conversions and scatter -> 139).
template <bool MAXIMA, bool DENSE = false>
__global__ void __launch_bounds__(RT_THREADS, 5)
row_topk_kernel(const __nv_bfloat16* __restrict__ H, long long ldh, int M, int N, int k,
                const float* __restrict__ gate, const uint8_t* __restrict__ alive, const float* __restrict__ maxima, long long ld_maxima, int vec,
                int* __restrict__ out_idx, float* __restrict__ out_val, __nv_bfloat16* __restrict__ dense) {
  pdl_wait();
  const int row = blockIdx.x;
  if (row >= M) return;
  const __nv_bfloat16* hrow = H + (long long)row * ldh;
  __nv_bfloat16* dense_row = DENSE ? dense + (size_t)row * N : nullptr;
  if constexpr (DENSE) {  // (N % 8 == 0; barriers lie between these and what is written over them)
    for (int c = threadIdx.x * 8; c < N; c += RT_THREADS * 8) *reinterpret_cast<uint4*>(dense_row + c) = make_uint4(0u, 0u, 0u, 0u);
  }
  __shared__ unsigned s_bits[RT_CAP];
  __shared__ int s_col[RT_CAP];
  __shared__ unsigned s_count[2][RT_WARPS];
  __shared__ int s_n, s_cursor, s_groups;
  constexpr int CAP = MAXIMA ? RT_CAP - RT_MAX_GROUPS : RT_CAP;
  bool use_radix = k > RT_BOUND_K;
  if (!use_radix) {
    if (threadIdx.x == 0) { s_n = 0; s_cursor = 0; s_groups = 0; }
    // ---- pass 1: maxima of this thread's eight column groups (non-positive values and NaN never enter)
    float mx[RT_MAXIMA];
#pragma unroll
    for (int i = 0; i < RT_MAXIMA; ++i) mx[i] = 0.0f;
    const float* groups = MAXIMA ? maxima + (long long)row * ld_maxima : nullptr;
    const int n_groups = (N + 31) / 32;
    if constexpr (MAXIMA) {
      for (int c0 = threadIdx.x; c0 < n_groups; c0 += RT_THREADS * RT_MAXIMA) {
#pragma unroll
        for (int i = 0; i < RT_MAXIMA; ++i)
          if (c0 + i * RT_THREADS < n_groups) mx[i] = fmaxf(mx[i], __ldg(groups + c0 + i * RT_THREADS));
      }
    } else {
#pragma unroll 4
      for (int c = threadIdx.x * 8; c < N; c += RT_THREADS * 8) {
        float v[8];
        gated_values8(hrow, gate, alive, c, N, vec != 0, v);
#pragma unroll
        for (int i = 0; i < 8; ++i) mx[i] = fmaxf(mx[i], v[i]);
      }
    }
    __syncthreads();
    unsigned mb[RT_MAXIMA];
#pragma unroll
    for (int i = 0; i < RT_MAXIMA; ++i) mb[i] = __float_as_uint(mx[i]);
    const unsigned bound = descend(mb, k, 16, s_count);
    // ---- pass 2: columns at or above the bound
    auto look_at = [&](int c, const float (&v)[8]) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const unsigned b = __float_as_uint(v[i]);
        if (v[i] > 0.0f && b >= bound) {
          const int pos = atomicAdd(&s_n, 1);
          if (pos < CAP) { s_bits[pos] = b; s_col[pos] = c + i; }
        }
      }
    };
    if constexpr (MAXIMA) {
      // the groups that reach the bound are listed first (in the columns' array, from its end), so that their reads go out together: four
      // lanes each
      int* s_group = s_col + RT_CAP - RT_MAX_GROUPS;
      for (int g = threadIdx.x; g < n_groups; g += RT_THREADS) {
        const float m = __ldg(groups + g);
        if (m > 0.0f ? __float_as_uint(m) >= bound : m != m) {  // (a NaN hides the others' maximum)
          const int pos = atomicAdd(&s_groups, 1);
          if (pos < RT_MAX_GROUPS) s_group[pos] = g;
        }
      }
      __syncthreads();
      const int n_list = s_groups;
      if (n_list <= RT_MAX_GROUPS) {
        const int sub = threadIdx.x & 3;
        for (int e0 = threadIdx.x >> 2; e0 < n_list; e0 += RT_THREADS / 4 * 2) {
          float v[2][8];
          int c[2];
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int e = e0 + i * (RT_THREADS / 4);
            c[i] = e < n_list ? s_group[e] * 32 + sub * 8 : N;
            if (c[i] < N) gated_values8(hrow, gate, alive, c[i], N, vec != 0, v[i]);
          }
#pragma unroll
          for (int i = 0; i < 2; ++i)
            if (c[i] < N) look_at(c[i], v[i]);
        }
      } else if (threadIdx.x == 0) {
        s_n = RT_CAP + 1;  // (values repeated thousands of times: the descent below)
      }
    } else {
#pragma unroll 2
      for (int c = threadIdx.x * 8; c < N; c += RT_THREADS * 8) {
        float v[8];
        gated_values8(hrow, gate, alive, c, N, vec != 0, v);
        look_at(c, v);
      }
    }
    __syncthreads();
    const int n_cand = s_n;
    use_radix = n_cand > CAP;  // (uniform)
    if (!use_radix) {
      // ---- the exact k-th value of the candidates
      unsigned thr = 0;
      if (n_cand > k) {
        unsigned mine[RT_CAP / RT_THREADS];
#pragma unroll
        for (int i = 0; i < RT_CAP / RT_THREADS; ++i) {
          const int j = threadIdx.x + i * RT_THREADS;
          mine[i] = j < n_cand ? s_bits[j] : 0u;
        }
        thr = descend(mine, k, 0, s_count);
      }
      // ---- winners: what lies above it first, then as many equal ones as there are places
      auto place = [&](int j) {
        const int pos = atomicAdd(&s_cursor, 1);
        if (pos < k) {
          const int c = s_col[j];
          const float v = __uint_as_float(s_bits[j]);
          const float a = gate != nullptr ? v / gate[c] : v;
          if constexpr (DENSE) {
            dense_row[c] = __float2bfloat16(a);
          } else {
            out_idx[(size_t)row * k + pos] = c;
            out_val[(size_t)row * k + pos] = a;
          }
        }
      };
      for (int j = threadIdx.x; j < n_cand; j += RT_THREADS)
        if (s_bits[j] > thr) place(j);
      __syncthreads();
      for (int j = threadIdx.x; j < n_cand; j += RT_THREADS)
        if (s_bits[j] == thr) place(j);
      for (int j = n_cand + threadIdx.x; j < k && !DENSE; j += RT_THREADS) {
        out_idx[(size_t)row * k + j] = -1;
        out_val[(size_t)row * k + j] = 0.0f;
      }
      return;
    }
  }
  row_topk_radix(hrow, row, N, k, gate, alive, out_idx, out_val, dense_row);
}

// Row top-k of stored pre-activations whose gated maxima per 32 columns are known, a warp per row (the encoder GEMM's epilogue leaves
// the maxima; T is how it stored the values). The rows of a batch are all in flight at once, and what a row takes is a short chain:
//   bound     512 groups of one or more neighbouring maxima at most, in registers: their k-th largest, 16 leading bits of it, which at
//             least k columns reach and with four times as many groups as codes few more do
//   groups    of 32 columns whose maximum reaches it, about k of them, listed in order; their columns, eight a lane
//   candidates above the bound listed in order; the exact k-th value of them; of equal ones the first columns
// Rows with more groups or candidates than there is room for (values repeated hundreds of times) are taken by the whole CTA afterwards, in
// the descent over the row that other kernels end in, too.
// As a CTA per row with barriers between the steps (row_topk_kernel<true>), 4096 rows of 32768 bf16, k 128, with a gate: 111 us; here 49
// (without: 135 and 53; 1024 rows: 46 and 37; 512 rows, where the chain is all there is: 29 and 36). 1024 rows of 16384 fp32, k 32: 20 us.
constexpr int RS_WARPS = 8, RS_PER = 16, RS_GROUPS = 256, RS_CAND = 384, RS_MAX_K = 128;
static_assert(RS_WARPS * 32 == RT_THREADS, "the fallback's CTA");
template <typename T>
__device__ __forceinline__ void stored_values8(const T* p, float (&v)[8]);
template <>
__device__ __forceinline__ void stored_values8<__nv_bfloat16>(const __nv_bfloat16* p, float (&v)[8]) {
  const uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
  const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
template <>
__device__ __forceinline__ void stored_values8<float>(const float* p, float (&v)[8]) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
// The largest t whose lowest `skip` bits are zero with count(key >= t) >= k over the warp, or (exactly = true) one that exactly k reach.
template <int N>
__device__ __forceinline__ unsigned warp_descend(const unsigned (&key)[N], int k, int skip, bool& exactly) {
  static_assert(N * 32 < 1024, "counts are packed in ten bits each");
  unsigned t = 0;
  exactly = false;
  for (int shift = 30; shift >= skip && !exactly; shift -= 2) {  // (bit 31 is never set)
    const unsigned t1 = t | (1u << shift), t2 = t | (2u << shift), t3 = t | (3u << shift);
    unsigned n = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) n += (unsigned)(key[i] >= t1) + ((unsigned)(key[i] >= t2) << 10) + ((unsigned)(key[i] >= t3) << 20);
    n = __reduce_add_sync(0xffffffffu, n);
    const int c1 = (int)(n & 1023u), c2 = (int)((n >> 10) & 1023u), c3 = (int)(n >> 20);
    if (c3 >= k) { t = t3; exactly = c3 == k; }
    else if (c2 >= k) { t = t2; exactly = c2 == k; }
    else if (c1 >= k) { t = t1; exactly = c1 == k; }
  }
  return t;
}

template <typename T>
__global__ void __launch_bounds__(RT_THREADS)
row_select_kernel(const T* __restrict__ H, long long ldh, const float* __restrict__ maxima, long long ld_maxima, int M, int N, int k,
                  const float* __restrict__ gate, int sorted, int* __restrict__ out_idx, float* __restrict__ out_val) {
  pdl_wait();
  __shared__ unsigned short s_group[RS_WARPS][RS_GROUPS];
  __shared__ unsigned s_key[RS_WARPS][RS_CAND];
  __shared__ int s_col[RS_WARPS][RS_CAND];
  __shared__ int s_full[RS_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned below = (1u << lane) - 1u;
  const int row = blockIdx.x * RS_WARPS + warp;
  if (lane == 0) s_full[warp] = 0;
  if (row < M) {
    const T* hrow = H + (long long)row * ldh;
    const float* mrow = maxima + (long long)row * ld_maxima;
    const int n_groups = (N + 31) / 32, fold = (n_groups + RS_PER * 32 - 1) / (RS_PER * 32);
    unsigned mx[RS_PER];
#pragma unroll
    for (int i = 0; i < RS_PER; ++i) mx[i] = 0u;  // (non-positive values and NaN never enter)
    for (int f = 0; f < fold; ++f) {
      float m[RS_PER];
#pragma unroll
      for (int i = 0; i < RS_PER; ++i) {
        const int g = (f * RS_PER + i) * 32 + lane;
        m[i] = g < n_groups ? __ldg(mrow + g) : 0.0f;
      }
#pragma unroll
      for (int i = 0; i < RS_PER; ++i) mx[i] = max(mx[i], __float_as_uint(fmaxf(m[i], 0.0f)) & 0x7fffffffu);
    }
    bool exactly;
    const unsigned bound = warp_descend(mx, k, 16, exactly);
    int n_list = 0;
    for (int g0 = 0; g0 < n_groups; g0 += 256) {
      float m[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) m[i] = g0 + i * 32 + lane < n_groups ? __ldg(mrow + g0 + i * 32 + lane) : 0.0f;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const bool hit = m[i] > 0.0f ? __float_as_uint(m[i]) >= bound : m[i] != m[i];  // (a NaN hides the others' maximum)
        const unsigned hits = __ballot_sync(0xffffffffu, hit);
        const int pos = n_list + __popc(hits & below);
        if (hit && pos < RS_GROUPS) s_group[warp][pos] = (unsigned short)(g0 + i * 32 + lane);
        n_list += __popc(hits);
      }
    }
    __syncwarp();
    int n_cand = n_list > RS_GROUPS ? RS_CAND + 1 : 0;
    if (n_list <= RS_GROUPS) {
      for (int e0 = 0; e0 < n_list; e0 += 16) {  // sixteen groups, four lanes each, two per lane in flight
        float v[2][8];
        int c[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int e = e0 + h * 8 + (lane >> 2);
          c[h] = e < n_list ? s_group[warp][e] * 32 + (lane & 3) * 8 : N;
          if (c[h] < N) {  // (N is a multiple of 8)
            stored_values8<T>(hrow + c[h], v[h]);
            if (gate != nullptr) {
              const float4 a = __ldg(reinterpret_cast<const float4*>(gate + c[h])), b = __ldg(reinterpret_cast<const float4*>(gate + c[h]) + 1);
              v[h][0] *= a.x; v[h][1] *= a.y; v[h][2] *= a.z; v[h][3] *= a.w;
              v[h][4] *= b.x; v[h][5] *= b.y; v[h][6] *= b.z; v[h][7] *= b.w;
            }
          } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[h][i] = 0.0f;
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          unsigned in = 0u;
#pragma unroll
          for (int i = 0; i < 8; ++i) in |= (v[h][i] > 0.0f && __float_as_uint(v[h][i]) >= bound) ? 1u << i : 0u;
          int inc = __popc(in);
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += a;
          }
          int pos = n_cand + inc - __popc(in);
          n_cand += __shfl_sync(0xffffffffu, inc, 31);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if ((in >> i) & 1u) {
              if (pos < RS_CAND) {
                s_key[warp][pos] = __float_as_uint(v[h][i]);
                s_col[warp][pos] = c[h] + i;
              }
              ++pos;
            }
          }
        }
      }
    }
    if (n_cand > RS_CAND) {
      if (lane == 0) s_full[warp] = 1;
    } else {
      __syncwarp();
      unsigned key[RS_CAND / 32];
#pragma unroll
      for (int i = 0; i < RS_CAND / 32; ++i) key[i] = i * 32 + lane < n_cand ? s_key[warp][i * 32 + lane] : 0u;
      unsigned t = 0;
      exactly = false;
      if (n_cand > k) t = warp_descend(key, k, 0, exactly);
      int above = 0;
#pragma unroll
      for (int i = 0; i < RS_CAND / 32; ++i) above += key[i] > t;
      const int ties_wanted = exactly ? k : t == 0u ? 0 : k - __reduce_add_sync(0xffffffffu, above);
      int n_win = 0, ties_seen = 0;
#pragma unroll
      for (int i = 0; i < RS_CAND / 32; ++i) {
        const bool eq = t != 0u && key[i] == t;
        const unsigned eqs = __ballot_sync(0xffffffffu, eq);
        const bool win = key[i] > t || (eq && ties_seen + __popc(eqs & below) < ties_wanted);
        const unsigned wins = __ballot_sync(0xffffffffu, win);
        const int col = win ? s_col[warp][i * 32 + lane] : 0;
        __syncwarp();
        if (win) {  // (to the front, at or before its own place)
          const int pos = n_win + __popc(wins & below);
          s_key[warp][pos] = key[i];
          s_col[warp][pos] = col;
        }
        n_win += __popc(wins);
        ties_seen += __popc(eqs);
        __syncwarp();
      }
      for (int w = lane; w < k; w += 32) {
        int place = w, col = -1;
        float val = 0.0f;
        if (w < n_win) {
          const unsigned u = s_key[warp][w];
          col = s_col[warp][w];
          val = __uint_as_float(u);
          if (gate != nullptr) val /= __ldg(gate + col);
          if (sorted) {
            place = 0;
#pragma unroll 8
            for (int j = 0; j < n_win; ++j) place += s_key[warp][j] + (j < w ? 1u : 0u) > u;
          }
        }
        out_idx[(size_t)row * k + place] = col;
        out_val[(size_t)row * k + place] = val;
      }
    }
  }
  __syncthreads();
  for (int w = 0; w < RS_WARPS; ++w) {
    const int r = blockIdx.x * RS_WARPS + w;
    if (s_full[w] != 0) {
      const T* hrow = H + (long long)r * ldh;
      int* idx = out_idx + (size_t)r * k;
      float* val = out_val + (size_t)r * k;
      row_topk_radix(hrow, r, N, k, gate, nullptr, out_idx, out_val);
      __syncthreads();
      // (which takes any of equal values, in any order) the first columns of the k-th value; values in descending order
      const int i = threadIdx.x;
      if (i < k) {
        s_col[0][i] = idx[i];
        s_key[0][i] = idx[i] >= 0 ? __float_as_uint(gated_value(hrow, gate, nullptr, idx[i])) : 0u;
      }
      __syncthreads();
      unsigned least = 0xffffffffu;
      for (int j = 0; j < k; ++j) least = min(least, s_key[0][j]);
      int n_above = 0;
      for (int j = 0; j < k; ++j) n_above += s_key[0][j] > least;
      if (least != 0u && warp == 0) {
        int n = 0;
        for (int c0 = 0; c0 < N && n < k - n_above; c0 += 256) {
          float v[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = c0 + j * 32 + lane < N ? gated_value(hrow, gate, nullptr, c0 + j * 32 + lane) : 0.0f;
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const bool eq = v[j] > 0.0f && __float_as_uint(v[j]) == least;
            const unsigned eqs = __ballot_sync(0xffffffffu, eq);
            const int pos = n + __popc(eqs & below);
            if (eq && pos < k - n_above) s_col[1][pos] = c0 + j * 32 + lane;
            n += __popc(eqs);
          }
        }
      }
      __syncthreads();
      if (i < k) {
        const unsigned u = s_key[0][i];
        const int col = s_col[0][i];
        if (u > least) {
          int place = 0;
          for (int j = 0; j < k; ++j) place += s_key[0][j] > u || (s_key[0][j] == u && s_col[0][j] < col);
          idx[place] = col;
          val[place] = gate != nullptr ? __uint_as_float(u) / gate[col] : __uint_as_float(u);
        }
        if (i < k - n_above) {
          const int c = least != 0u ? s_col[1][i] : -1;
          idx[n_above + i] = c;
          val[n_above + i] = c < 0 ? 0.0f : gate != nullptr ? __uint_as_float(least) / gate[c] : __uint_as_float(least);
        }
      }
      __syncthreads();
    }
  }
}

int row_select_max_k() { return RS_MAX_K; }

int row_select_launch(const __nv_bfloat16* H16, const float* H32, long long ldh, const float* maxima, long long ld_maxima, int M, int N, int k,
                      const float* gate, int sorted, int* out_idx, float* out_val, cudaStream_t stream) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(H16) | reinterpret_cast<uintptr_t>(H32) | reinterpret_cast<uintptr_t>(gate);
  if ((H16 != nullptr) == (H32 != nullptr) || k < 1 || k > RS_MAX_K || N % 8 != 0 || N > 65535 * 32 || ldh % 8 != 0 || at % 16 != 0) return (int)cudaErrorInvalidValue;
  if (M <= 0) return 0;
  const int blocks = (M + RS_WARPS - 1) / RS_WARPS;
  if (H16 != nullptr) launch(row_select_kernel<__nv_bfloat16>, blocks, RT_THREADS, 0, stream, H16, ldh, maxima, ld_maxima, M, N, k, gate, sorted, out_idx, out_val);
  else launch(row_select_kernel<float>, blocks, RT_THREADS, 0, stream, H32, ldh, maxima, ld_maxima, M, N, k, gate, sorted, out_idx, out_val);
  return (int)cudaGetLastError();
}

int row_topk_launch(const __nv_bfloat16* H, long long ldh, int M, int N, int k, const float* gate,
                    const uint8_t* alive, const float* maxima, long long ld_maxima, int* out_idx, float* out_val, cudaStream_t stream) {
  const bool vec = N % 8 == 0 && ldh % 8 == 0 && reinterpret_cast<uintptr_t>(H) % 16 == 0 && reinterpret_cast<uintptr_t>(gate) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(alive) % 8 == 0;
  if (maxima != nullptr) launch(row_topk_kernel<true>, M, RT_THREADS, 0, stream, H, ldh, M, N, k, gate, alive, maxima, ld_maxima, vec ? 1 : 0, out_idx, out_val, nullptr);
  else launch(row_topk_kernel<false>, M, RT_THREADS, 0, stream, H, ldh, M, N, k, gate, alive, nullptr, 0, vec ? 1 : 0, out_idx, out_val, nullptr);
  return (int)cudaGetLastError();
}

int row_topk_dense_launch(const __nv_bfloat16* H, int M, int N, int k, const float* gate, __nv_bfloat16* dense, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (N % 8 != 0 || (reinterpret_cast<uintptr_t>(dense) & 15) != 0) return (int)cudaErrorInvalidValue;
  const bool vec = ((reinterpret_cast<uintptr_t>(H) | reinterpret_cast<uintptr_t>(gate)) & 15) == 0;
  return (int)launch(row_topk_kernel<false, true>, M, RT_THREADS, 0, stream, H, N, M, N, k, gate, nullptr, nullptr, 0, vec ? 1 : 0, nullptr, nullptr, dense);
}

// ------------------------------------------------------------------------------------------------
// TopK activation on fp32 pre-activations, dense in and dense out:  out = topk(relu(g)) / norm  with  g = (h + bias) * norm  (bias and
// norm optional), k entries per row; of equal values the first columns. One CTA per row: group maxima bound the k-th value, a second
// pass (from L1 / L2) writes the row's zeros and collects the few entries at or above the bound, and the k best of them are written
// over the zeros. Bound by reading h and writing out. 4096 x 24576, k 50, bias, gate, selection, mask and division: 3.2 ms as torch
// operations -> 319 us.
// The arithmetic is that of the operations it replaces, element by element (subnormals included: no flush to zero): NaN and -inf (which
// relu(x) = x * [x > 0] turns into NaN) rank first and stay NaN everywhere, an unselected +inf becomes NaN, and so does everything over a
// norm of 0 or NaN.
//
// ESTIMATE: there is no h, only lower ends of g in bf16 (fp32_gemm.cu, which says what they enclose). What is selected, and the selected
// values, are those of the fp32 sum x . W^T in ascending order of k with one rounding per term.
//   The k-th largest of the group maxima of the lower ends is reached by at least k columns, and whatever is selected has its upper end
// at or above it. The upper end is the lower one plus what rounding it down to bf16 may have taken (2^-7 of it) plus twice the bound on the
// estimate's error. Where that is small against the k-th end (a 64th) for the column where it is largest, all columns take that one's, and
// neither pass reads anything per column but the ends; elsewhere (a few features of large norm, long rows, few positive values) the second pass
// reads every column's own: 4096 x 24576 x 768, k 50, at a hundredth 660 us with the largest for all and 664 with each its own, at a fiftieth 698
// and 660, at a 36th 722 and 661. (2048 x 24576 x 4096 with one row of W thirty times the others: 11.3 ms with the largest for all, 1.66 so.)
// The columns that may be selected (k and a few) are summed up in order before the exact selection.
//   Columns that the bound says nothing about (their lower end is NaN) are among them; rows with more such columns than there is room for,
// and all rows where the product gave up, are listed, multiplied in order as a whole (rows_product.cu) and selected from exactly. All
// decisions are taken on the device.
//   With ends from one fp16 product (topk_narrow_launch) the bound and the columns come from the maxima of 32 columns, and the ends are
// read only in groups that may hold something. Rows with more than 256 + 4 k columns in question are listed instead of summed up; where they are more
// than an eighth of all rows, three bf16 products propose for the whole batch again, and the listed rows are selected from in the form above
// (topk_wide_launch). Elsewhere the kernels of that second proposal leave at once, 15 us in all.
// 4096 x 24576 x 768, k 50: lower ends of three products, each row's read twice, 286 us; by maxima of those of one product 267, and 255
// since the zeros (403 MB) leave while the bound is worked out. The rest are the rows of W, 3 kB for each of about 60 columns. Twelve rows of W at a time per warp take one
// pass over those columns where eight take two (387 us with 72 columns a row).
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned topk_key(float g) {
  const unsigned b = __float_as_uint(g);
  if ((b & 0x7fffffffu) > 0x7f800000u || b == 0xff800000u) return 0x7fffffffu;
  return (int)b > 0 ? b : 0u;
}
__device__ __forceinline__ bool below(float a, float b) {  // a < b: false for a NaN, subnormals as they are
  int r;
  asm("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %1, %2;\n\tselp.s32 %0, 1, 0, p;\n\t}" : "=r"(r) : "f"(a), "f"(b));
  return r != 0;
}
__device__ __forceinline__ bool not_finite(float x) { return (__float_as_uint(x) & 0x7fffffffu) >= 0x7f800000u; }

struct TopkDenseParams {
  const float* h;
  const __nv_bfloat16* lo;  // ESTIMATE: [B, N] lower ends, and with them
  const float* x;           // [B, K] and [N, K]
  const float* W;
  const float* xn;          // [B] 2-norms (fp32_gemm.cu)
  const uint32_t* top;      // the largest error bound of a column over rel * xn; whether a norm is 0 or NaN; from the fifth word on every column's bound, bf16
  const int* status;        // of the product
  float rel;                // the bound's factor (with lost: half_rel's), and another one where wide[0] > wide_limit
  const float* lost;
  float rel_wide;
  const int* wide;          // [0] number of rows, then which
  int wide_limit;
  int most;                 // entries of a row to be summed up at most
  const float* maxima;      // MAXIMA: [B][ld_maxima] the ends' group_max of 32 columns each
  long long ld_maxima;
  int K;
  int* todo;        // ESTIMATE: [1 + B] number of rows left over, and which
  const int* rows;  // or the rows to work on, in this form
  const float* bias;
  const float* norm;
  float* out;
  int N, k;
  bool vec;
};

// g of columns [c, c + 4) and the norms (columns past the end: 0 and 1)
__device__ __forceinline__ void topk_dense_load(const TopkDenseParams& p, const float* __restrict__ h, int c, float (&g)[4], float (&n)[4]) {
  float b[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int i = 0; i < 4; ++i) n[i] = 1.0f;
  if (p.vec) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(h + c));
    g[0] = a.x; g[1] = a.y; g[2] = a.z; g[3] = a.w;
    if (p.bias != nullptr) {
      const float4 t = __ldg(reinterpret_cast<const float4*>(p.bias + c));
      b[0] = t.x; b[1] = t.y; b[2] = t.z; b[3] = t.w;
    }
    if (p.norm != nullptr) {
      const float4 t = __ldg(reinterpret_cast<const float4*>(p.norm + c));
      n[0] = t.x; n[1] = t.y; n[2] = t.z; n[3] = t.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool in = c + i < p.N;
      g[i] = in ? __ldg(h + c + i) : 0.0f;
      if (in && p.bias != nullptr) b[i] = p.bias[c + i];
      if (in && p.norm != nullptr) n[i] = p.norm[c + i];
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (p.bias != nullptr) g[i] = add_rn(g[i], b[i]);
    if (p.norm != nullptr) g[i] = mul_rn(g[i], n[i]);
  }
}

// Lower ends of columns [c, c + 8) (past the end: -1, which neither reaches a bound nor enters)
__device__ __forceinline__ void topk_ends_load(const TopkDenseParams& p, const __nv_bfloat16* __restrict__ lo, int c, float (&g)[8]) {
  if (p.vec) {
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(lo + c));
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      g[2 * i] = __uint_as_float(w[i] << 16);
      g[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) g[i] = c + i < p.N ? __bfloat162float(lo[c + i]) : -1.0f;
  }
}

// x . W[cols[j]], fp32, in ascending order (K % 4 == 0) for j < n: done(j, sum). A sum is one thread's chain of K roundings, but its row
// of W is fetched by the whole warp: pieces of 32 columns of eight candidates' rows and of x are copied to shared memory, whole
// sectors a row, one piece ahead. (Each thread reading its own row, 16 bytes at a time, kept the L1 cache busy with a line per thread and
// load: 373 us for the whole selection.) Neighbouring candidates go to different warps.
constexpr int DOT_K = 32, DOT_PITCH = DOT_K + 4;  // (the pitch: eight rows' 16-byte pieces in different banks)
template <int DOT_ROWS>
struct DotTiles { float w[RT_WARPS][2][DOT_ROWS + 1][DOT_PITCH]; };
template <int DOT_ROWS, class Done>
__device__ __forceinline__ void dots_in_order(DotTiles<DOT_ROWS>& tiles, const float* __restrict__ x, const float* __restrict__ W, int K, const int* cols, int n, Done&& done) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int PIECES = (DOT_ROWS + 1) * DOT_K / 4, PER_LANE = (PIECES + 31) / 32;
  for (int base = warp; base < n; base += DOT_ROWS * RT_WARPS) {
    const int rows = min(DOT_ROWS, (n - base + RT_WARPS - 1) / RT_WARPS);  // candidates base + r * RT_WARPS
    const float* src[PER_LANE];
    int at[PER_LANE];  // column within the piece, -1: nothing to fetch
#pragma unroll
    for (int i = 0; i < PER_LANE; ++i) {
      const int e = i * 32 + lane, r = e / (DOT_K / 4);
      at[i] = r < rows || r == DOT_ROWS ? (e % (DOT_K / 4)) * 4 : -1;
      src[i] = r < rows ? W + (size_t)cols[base + r * RT_WARPS] * K : x;
    }
    auto fetch = [&](int k0, int buf) {
#pragma unroll
      for (int i = 0; i < PER_LANE; ++i) {
        const int r = (i * 32 + lane) / (DOT_K / 4);
        if (at[i] >= 0 && k0 + at[i] < K)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(&tiles.w[warp][buf][r][at[i]])), "l"(src[i] + k0 + at[i]) : "memory");
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float s = 0.0f;
    fetch(0, 0);
    for (int k0 = 0, buf = 0; k0 < K; k0 += DOT_K, buf ^= 1) {
      fetch(k0 + DOT_K, buf ^ 1);  // (past the end: an empty group)
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
      if (lane < rows) {
        const float4* a = reinterpret_cast<const float4*>(tiles.w[warp][buf][DOT_ROWS]);
        const float4* b = reinterpret_cast<const float4*>(tiles.w[warp][buf][lane]);
        if (k0 + DOT_K <= K) {
#pragma unroll
          for (int i = 0; i < DOT_K / 4; ++i) {
            s = fma_rn(a[i].x, b[i].x, s);
            s = fma_rn(a[i].y, b[i].y, s);
            s = fma_rn(a[i].z, b[i].z, s);
            s = fma_rn(a[i].w, b[i].w, s);
          }
        } else {
          for (int i = 0; i < (K - k0) / 4; ++i) {
            s = fma_rn(a[i].x, b[i].x, s);
            s = fma_rn(a[i].y, b[i].y, s);
            s = fma_rn(a[i].z, b[i].z, s);
            s = fma_rn(a[i].w, b[i].w, s);
          }
        }
      }
      __syncwarp();  // (the buffer is filled again in the next turn)
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (lane < rows) done(base + lane * RT_WARPS, s);
  }
}

// Sum over the CTA, the same in every thread.
__device__ __forceinline__ int cta_count(int mine, unsigned (&words)[RT_WARPS]) {
  const unsigned total = __reduce_add_sync(0xffffffffu, (unsigned)mine);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) words[threadIdx.x >> 5] = total;
  __syncthreads();
  return (int)__reduce_add_sync(0xffffffffu, (threadIdx.x & 31) < RT_WARPS ? words[threadIdx.x & 31] : 0u);
}

template <bool ESTIMATE, int CAP = RT_CAP, int DOT_ROWS = 8, bool MAXIMA = false>
__device__ __forceinline__ void topk_dense_row(const TopkDenseParams& p, int row) {
  __shared__ unsigned s_key[CAP];
  __shared__ int s_col[CAP];
  __shared__ unsigned s_count[2][RT_WARPS];
  __shared__ int s_n, s_above, s_equal;
  const float* h = ESTIMATE ? nullptr : p.h + (size_t)row * p.N;
  const __nv_bfloat16* lo = ESTIMATE ? p.lo + (size_t)row * p.N : nullptr;
  float* out = p.out + (size_t)row * p.N;
  const int N = p.N, k = p.k;
  if (ESTIMATE && p.status[0] != 0) {  // there are no ends
    if (threadIdx.x == 0) p.todo[1 + atomicAdd(p.todo, 1)] = row;
    return;
  }
  if (threadIdx.x == 0) { s_n = 0; s_above = 0; s_equal = 0; }
  unsigned mx[RT_MAXIMA];
#pragma unroll
  for (int i = 0; i < RT_MAXIMA; ++i) mx[i] = 0u;
  const float* maxima = MAXIMA ? p.maxima + row * p.ld_maxima : nullptr;
  const int groups = MAXIMA ? (int)p.ld_maxima : 0;
  if constexpr (MAXIMA) {
    for (int c = threadIdx.x * 4; c < groups; c += RT_THREADS * 4) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(maxima + c));
      const float g[4] = {v.x, v.y, v.z, v.w};
      const int h4 = c / (RT_THREADS * 4) & 1 ? 4 : 0;  // (up to 2048 groups: each by itself)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const unsigned b = __float_as_uint(g[i]) & 0xffff0000u;
        if (h4 == 0) mx[i] = max(mx[i], b);
        else mx[4 + i] = max(mx[4 + i], b);
      }
    }
  } else if constexpr (ESTIMATE) {
#pragma unroll 4
    for (int c = threadIdx.x * 8; c < N; c += RT_THREADS * 8) {
      float g[8];
      topk_ends_load(p, lo, c, g);
#pragma unroll
      for (int i = 0; i < 8; ++i) mx[i] = __float_as_uint(fmaxf(__uint_as_float(mx[i]), g[i]));  // (a NaN does not enter)
    }
  } else {
#pragma unroll 2
    for (int c = threadIdx.x * 8; c < N; c += RT_THREADS * 8) {
#pragma unroll
      for (int half = 0; half < 8; half += 4) {
        if (c + half >= N) break;
        float g[4], nm[4];
        topk_dense_load(p, h, c + half, g, nm);
#pragma unroll
        for (int i = 0; i < 4; ++i) mx[half + i] = max(mx[half + i], topk_key(g[i]));
      }
    }
  }
  const float nan = __uint_as_float(0x7fffffffu);
  // the row's zeros (NaN over a norm of 0 or NaN) for columns [c, c + 8)
  auto clear = [&](int c, bool any_bad) {
    float z[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) z[i] = 0.0f;
    if (any_bad) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const unsigned nb = c + i < N ? __float_as_uint(p.norm[c + i]) & 0x7fffffffu : 1u;
        if (nb == 0u || nb > 0x7f800000u) z[i] = nan;
      }
    }
    if (p.vec) {
      __stcs(reinterpret_cast<float4*>(out + c), make_float4(z[0], z[1], z[2], z[3]));
      __stcs(reinterpret_cast<float4*>(out + c + 4), make_float4(z[4], z[5], z[6], z[7]));
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (c + i < N) out[c + i] = z[i];
    }
  };
  if constexpr (MAXIMA) {  // (they leave while the bound is worked out)
    const bool any_bad = p.top[1] != 0u;
    for (int c = threadIdx.x * 8; c < N; c += RT_THREADS * 8) clear(c, any_bad);
  }
  unsigned thr = descend(mx, k, 16, s_count);  // a bound until the exact value is known (0: fewer than k positive maxima)
  auto enter = [&](int c, unsigned key) {
    const int pos = atomicAdd(&s_n, 1);
    if (pos < CAP) { s_key[pos] = key; s_col[pos] = c; }
  };
  if constexpr (ESTIMATE) {
    // (16 units of 2^-24 more for the roundings of the ends; the last term for lower ends that are subnormal)
    const float rel = p.wide != nullptr && p.wide[0] > p.wide_limit ? p.rel_wide : p.lost != nullptr ? half_rel(p.rel, p.lost[row], p.top + 2) : p.rel;
    const float width = mul_up(2.0f * (rel + 1e-6f), p.xn[row]);
    const float room = add_rn(mul_up(width, __uint_as_float(p.top[0])), 1e-37f);
    const float thr_f = __uint_as_float(max(thr, 1u));
    const __nv_bfloat16* widths = below(mul_rn(room, 64.0f), thr_f) ? nullptr : reinterpret_cast<const __nv_bfloat16*>(p.top + 4);
    const bool any_bad = p.top[1] != 0u;
    auto visit = [&](int c) {  // columns [c, c + 8)
      float g[8], r[8];
      topk_ends_load(p, lo, c, g);
#pragma unroll
      for (int i = 0; i < 8; ++i) r[i] = room;
      if (widths != nullptr) {
        topk_ends_load(p, widths, c, r);
#pragma unroll
        for (int i = 0; i < 8; ++i) r[i] = add_rn(mul_up(width, r[i]), 1e-37f);
      }
      unsigned in = 0u;
#pragma unroll
      for (int i = 0; i < 8; ++i) in |= below(add_rn(fma_rn(fabsf(g[i]), 0.0079f, g[i]), r[i]), thr_f) ? 0u : 1u << i;  // (a NaN enters)
      while (in != 0u) {
        const int i = __ffs(in) - 1;
        in &= in - 1u;
        if (c + i < N) enter(c + i, 0u);
      }
    };
    const bool by_groups = MAXIMA && widths == nullptr;
    if (by_groups) {  // only the groups that may hold something (a lane of a group's four: eight of its columns)
      for (int base = (int)(threadIdx.x >> 5) * 32; base < groups; base += RT_THREADS) {
        const int j = base + (int)(threadIdx.x & 31);
        unsigned b = 0u;
        bool in = false;
        if (j < groups) {
          b = __float_as_uint(__ldg(maxima + j));
          const float g = __uint_as_float(b & 0xffff0000u);
          in = (b & 1u) != 0u || !below(add_rn(fma_rn(g, 0.0079f, g), room), thr_f);
        }
        unsigned mask = __ballot_sync(0xffffffffu, in);
        while (mask != 0u) {  // eight groups at a time
          unsigned mine = mask;
          for (int s = (int)(threadIdx.x & 31) >> 2; s > 0 && mine != 0u; --s) mine &= mine - 1u;
          if (mine != 0u) {
            const int c = (base + __ffs(mine) - 1) * 32 + ((int)threadIdx.x & 3) * 8;
            if (c < N) visit(c);
          }
          for (int s = 0; s < 8 && mask != 0u; ++s) mask &= mask - 1u;
        }
      }
    }
    if (!by_groups) {
#pragma unroll 2
      for (int c = threadIdx.x * 8; c < N; c += RT_THREADS * 8) {
        visit(c);
        if constexpr (!MAXIMA) clear(c, any_bad);
      }
    }
  } else {
#pragma unroll 2
    for (int c = threadIdx.x * 8; c < N; c += RT_THREADS * 8) {
#pragma unroll
      for (int half = 0; half < 8; half += 4) {
        if (c + half >= N) break;
        float g[4], nm[4];
        topk_dense_load(p, h, c + half, g, nm);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const unsigned nb = __float_as_uint(nm[i]) & 0x7fffffffu;
          const unsigned key = topk_key(g[i]);
          if (key != 0u && key >= thr) enter(c + half + i, key);
          g[i] = nb == 0u || nb > 0x7f800000u || not_finite(g[i]) ? nan : 0.0f;
        }
        if (p.vec) {
          __stcs(reinterpret_cast<float4*>(out + c + half), make_float4(g[0], g[1], g[2], g[3]));
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (c + half + i < N) out[c + half + i] = g[i];
        }
      }
    }
  }
  __syncthreads();  // (also: the zeros are written before what is written over them)
  const int n = s_n;
  if constexpr (ESTIMATE) {
    if (n > p.most) {
      if (threadIdx.x == 0) p.todo[1 + atomicAdd(p.todo, 1)] = row;
      return;
    }
    __shared__ __align__(16) DotTiles<DOT_ROWS> tiles;
    dots_in_order(tiles, p.x + (size_t)row * p.K, p.W, p.K, s_col, n, [&](int j, float g) {
      const int c = s_col[j];
      if (p.bias != nullptr) g = add_rn(g, p.bias[c]);
      unsigned nb = 1u;
      if (p.norm != nullptr) {
        g = mul_rn(g, p.norm[c]);
        nb = __float_as_uint(p.norm[c]) & 0x7fffffffu;
      }
      s_key[j] = topk_key(g);
      if (not_finite(g) || nb == 0u || nb > 0x7f800000u) out[c] = nan;  // (the last two are NaN already)
    });
    __syncthreads();
  }
  auto put = [&](int c, unsigned key) {
    if (key == 0x7fffffffu) return;  // (what is NaN already stays so)
    float v = __uint_as_float(key);
    if (p.norm != nullptr) v = div_rn(v, p.norm[c]);
    out[c] = v;
  };
  if (n <= CAP) {
    if (n > k) {
      unsigned mine[CAP / RT_THREADS];
#pragma unroll
      for (int i = 0; i < CAP / RT_THREADS; ++i) {
        const int j = threadIdx.x + i * RT_THREADS;
        mine[i] = j < n ? s_key[j] : 0u;
      }
      thr = descend(mine, k, 0, s_count);
    } else {
      thr = 0u;
    }
    for (int j = threadIdx.x; j < n; j += RT_THREADS) {
      const unsigned key = s_key[j];
      if (key > thr) {
        put(s_col[j], key);
        if (thr != 0u) atomicAdd(&s_above, 1);
      } else if (key == thr && thr != 0u) {
        atomicAdd(&s_equal, 1);
      }
    }
    if (thr == 0u) return;  // (all of them)
    __syncthreads();
    const int places = k - s_above;
    const bool all = s_equal <= places;
    for (int j = threadIdx.x; j < n; j += RT_THREADS) {
      if (s_key[j] != thr) continue;
      const int c = s_col[j];
      int before = 0;
      if (!all)
        for (int i = 0; i < n; ++i) before += s_key[i] == thr && s_col[i] < c;
      if (before < places) put(c, thr);
    }
    return;
  }
  if constexpr (!ESTIMATE) {
    // values repeated thousands of times: the descent over the row itself, one pass per bit
    auto keys_of = [&](auto&& visit) {
      for (int c = threadIdx.x * 4; c < N; c += RT_THREADS * 4) {
        float g[4], nm[4];
        topk_dense_load(p, h, c, g, nm);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const unsigned key = topk_key(g[i]);
          if (key != 0u) visit(c + i, key);
        }
      }
    };
    auto count_of = [&](auto&& which) {
      int mine = 0;
      keys_of([&](int c, unsigned key) { mine += which(c, key); });
      return cta_count(mine, s_count[0]);
    };
    thr = 0u;
    for (int bit = 30; bit >= 0; --bit) {
      const unsigned trial = thr | (1u << bit);
      if (count_of([&](int, unsigned key) { return key >= trial; }) >= k) thr = trial;
    }
    keys_of([&](int c, unsigned key) { if (key > thr) put(c, key); });
    if (thr == 0u || thr == 0x7fffffffu) return;
    // the equal ones up to the column at which the places are taken
    const int places = k - count_of([&](int, unsigned key) { return key > thr; });
    int end = 0;  // at most `places` equal values lie in columns below it
    for (int bit = 30; bit >= 0; --bit) {
      const long long trial = (long long)end + (1LL << bit);
      if (trial <= N && count_of([&](int c, unsigned key) { return key == thr && c < trial; }) <= places) end = (int)trial;
    }
    keys_of([&](int c, unsigned key) { if (key == thr && c < end) put(c, thr); });
  }
}

template <bool ESTIMATE, int CAP = RT_CAP, int DOT_ROWS = 8, bool MAXIMA = false>
__global__ void __launch_bounds__(RT_THREADS, 5)
topk_dense_kernel(const TopkDenseParams p) {
  pdl_wait();
  topk_dense_row<ESTIMATE, CAP, DOT_ROWS, MAXIMA>(p, blockIdx.x);
}

__global__ void __launch_bounds__(RT_THREADS, 5)
topk_wide_kernel(const TopkDenseParams p) {
  pdl_wait();
  const int n = p.wide[0];
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    topk_dense_row<true>(p, p.wide[1 + i]);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(RT_THREADS, 5)
topk_dense_rows_kernel(const TopkDenseParams p) {
  pdl_wait();
  const int n = p.rows[0];
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    topk_dense_row<false>(p, p.rows[1 + i]);
    __syncthreads();
  }
}

int topk_dense_launch(const float* h, const float* bias, const float* norm, int B, int N, int k, float* out, cudaStream_t stream) {
  if (B <= 0 || N <= 0) return 0;
  if (k < 1 || k > RT_BOUND_K) return (int)cudaErrorInvalidValue;
  TopkDenseParams p = {};
  p.h = h; p.bias = bias; p.norm = norm; p.out = out; p.N = N; p.k = k;
  p.vec = N % 4 == 0 && ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(norm) |
                          reinterpret_cast<uintptr_t>(out)) % 16 == 0);
  launch(topk_dense_kernel<false>, B, RT_THREADS, 0, stream, p);
  return (int)cudaGetLastError();
}

constexpr int NARROW_CAP = 4 * RT_THREADS;  // (what it leaves of the shared memory holds more rows of W at a time)

static bool estimate_args_fit(const float* x, const float* W, int K, int k) {
  return k >= 1 && k <= RT_BOUND_K && K >= 1 && K <= kEstimateMaxK && K % 4 == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(W)) & 15) == 0;
}

// The rows listed in todo: their products in order, and the selection from those.
static int finish_rows(TopkDenseParams p, float* h, int B, int* todo, cudaStream_t stream) {
  RowsProductParams r = {};
  r.A = p.x; r.B = p.W; r.C = h; r.N = p.N; r.K = p.K; r.rows = todo; r.max_rows = B;
  const int e = rows_product_launch(r, false, stream);
  if (e != 0) return e;
  p.rows = todo;
  p.h = h;
  p.vec = p.N % 4 == 0 && ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(p.bias) | reinterpret_cast<uintptr_t>(p.norm) |
                            reinterpret_cast<uintptr_t>(p.out)) % 16 == 0);
  return (int)launch(topk_dense_rows_kernel, B < 148 * 5 ? B : 148 * 5, RT_THREADS, 0, stream, p);
}

// The same with lower ends `lo` from an estimate of x W^T; h: fp32 [B, N] for the products of rows that are left over (it may share
// memory with lo, which is no longer read then). todo: int [1 + B], todo[0] zeroed.
int topk_estimate_launch(const __nv_bfloat16* lo, float* h, const float* x, const float* W, const float* xn, const uint32_t* top, int K, const float* bias,
                         const float* norm, int B, int N, int k, const int* status, int* todo, float* out, cudaStream_t stream) {
  if (B <= 0 || N <= 0) return 0;
  if (!estimate_args_fit(x, W, K, k)) return (int)cudaErrorInvalidValue;
  TopkDenseParams p = {};
  p.lo = lo; p.x = x; p.W = W; p.xn = xn; p.top = top; p.status = status; p.K = K; p.todo = todo; p.bias = bias; p.norm = norm; p.out = out; p.N = N; p.k = k;
  p.rel = estimate_rel(K);
  p.most = RT_CAP;
  p.vec = N % 8 == 0 && ((reinterpret_cast<uintptr_t>(lo) | reinterpret_cast<uintptr_t>(out)) % 16 == 0);
  const cudaError_t e = launch(topk_dense_kernel<true>, B, RT_THREADS, 0, stream, p);
  return e != cudaSuccess ? (int)e : finish_rows(p, h, B, todo, stream);
}

// With lower ends from one fp16 product (half_ends_launch): what can be decided by them without summing up more than a few times k entries of a
// row. The other rows go to the list `wide`, int [1 + B], wide[0] zeroed.
int topk_narrow_launch(const __nv_bfloat16* lo, const float* maxima, long long ld_maxima, const float* x, const float* W, const float* xn, const float* lost, const uint32_t* top, int K, const float* bias, const float* norm,
                       int B, int N, int k, const int* status, int* wide, float* out, cudaStream_t stream) {
  if (B <= 0 || N <= 0) return 0;
  if (!estimate_args_fit(x, W, K, k) || maxima == nullptr || ld_maxima % 4 != 0 || (reinterpret_cast<uintptr_t>(maxima) & 15) != 0) return (int)cudaErrorInvalidValue;
  TopkDenseParams p = {};
  p.lo = lo; p.x = x; p.W = W; p.xn = xn; p.top = top; p.status = status; p.K = K; p.todo = wide; p.bias = bias; p.norm = norm; p.out = out; p.N = N; p.k = k;
  p.rel = estimate_rel_half(K);
  p.lost = lost;
  p.maxima = maxima; p.ld_maxima = ld_maxima;
  p.most = min(256 + 4 * k, RT_CAP);
  p.vec = N % 8 == 0 && ((reinterpret_cast<uintptr_t>(lo) | reinterpret_cast<uintptr_t>(out)) % 16 == 0);
  return (int)(p.most <= NARROW_CAP ? launch(topk_dense_kernel<true, NARROW_CAP, 12, true>, B, RT_THREADS, 0, stream, p)
                                         : launch(topk_dense_kernel<true, RT_CAP, 8, true>, B, RT_THREADS, 0, stream, p));
}

// The rows of that list, with lower ends from three products where they are more than wide_limit (lo holds those then), and from one elsewhere.
int topk_wide_launch(const __nv_bfloat16* lo, float* h, const float* x, const float* W, const float* xn, const float* lost, const uint32_t* top, int K, const float* bias,
                     const float* norm, int B, int N, int k, const int* status, const int* wide, int wide_limit, int* todo, float* out, cudaStream_t stream) {
  if (B <= 0 || N <= 0) return 0;
  if (!estimate_args_fit(x, W, K, k)) return (int)cudaErrorInvalidValue;
  TopkDenseParams p = {};
  p.lo = lo; p.x = x; p.W = W; p.xn = xn; p.top = top; p.status = status; p.K = K; p.todo = todo; p.bias = bias; p.norm = norm; p.out = out; p.N = N; p.k = k;
  p.rel = estimate_rel_half(K);
  p.lost = lost;
  p.rel_wide = estimate_rel(K);
  p.wide = wide;
  p.wide_limit = wide_limit;
  p.most = RT_CAP;
  p.vec = N % 8 == 0 && ((reinterpret_cast<uintptr_t>(lo) | reinterpret_cast<uintptr_t>(out)) % 16 == 0);
  const cudaError_t e = launch(topk_wide_kernel, B < 148 * 5 ? B : 148 * 5, RT_THREADS, 0, stream, p);
  return e != cudaSuccess ? (int)e : finish_rows(p, h, B, todo, stream);
}

}  // namespace lmsae
