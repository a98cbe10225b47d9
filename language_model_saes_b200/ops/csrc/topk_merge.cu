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

namespace lmsae {

constexpr int MERGE_WARPS = 4;

// One warp per row. Positive floats order like their bit patterns, so the k-th largest candidate is found by a
// descent over the 31 value bits (count(key >= t) per trial, one warp reduction each) instead of ranking every
// candidate against every other one; candidates equal to the threshold get the remaining places in slot order. The
// (at most k) winners are compacted into shared memory and ranked among themselves. Only winners whose candidate
// slot lies in [own_lo, own_hi) are written, in value-descending order FROM SLOT 0 ON (the rest of the row is
// (-1, 0)): consumers of a shard's codes may stop at the first empty slot.
//
// comm.mode selects what surrounds the merge under feature sharding:
//   kMergeLocal  nothing (single GPU, or lists that are exchanged by other means)
//   kMergePush   the row's k (value, column) pairs are not written to out_* but stored straight into segment
//                [rank * k, (rank + 1) * k) of EVERY rank's merge input (the all-gather of the candidate lists by
//                peer stores, fused into the kernel that produces them); the last block publishes the epoch
//   kMergeWait   the kernel first waits (bounded) until every rank has published the epoch for the candidate
//                phase, then merges the gathered lists it finds in this rank's own buffer
__global__ void __launch_bounds__(MERGE_WARPS * 32)
topk_merge_kernel(const float* cand_val, const int* cand_idx, int M, int C, int k,  // may be peer-written: no read-only path
                  const float* __restrict__ gate, int own_lo, int own_hi, int emit_gated,
                  int* __restrict__ out_idx, float* __restrict__ out_val, const MergeComm comm) {
  extern __shared__ uint8_t smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  // per warp: keys[C], ids[C], winner keys[k], winner slots[k], staged output ids[k] and values[k]
  uint32_t* skey = reinterpret_cast<uint32_t*>(smem_raw) + (size_t)warp * (2 * C + 4 * k);
  int* sidx = reinterpret_cast<int*>(skey + C);
  uint32_t* wkey = reinterpret_cast<uint32_t*>(sidx + C);
  int* wslot = reinterpret_cast<int*>(wkey + k);
  int* oidx = wslot + k;
  float* oval = reinterpret_cast<float*>(oidx + k);

  bool inputs_ok = true;
  if (comm.mode == kMergeWait) inputs_ok = wait_all_sources(comm.pt, kPhaseCand, comm.epoch, comm.status);

  for (int row = blockIdx.x * MERGE_WARPS + warp; row < M; row += gridDim.x * MERGE_WARPS) {
    for (int i = lane; i < k; i += 32) {
      oidx[i] = -1;
      oval[i] = 0.0f;
    }
    if (inputs_ok) {
      const float* cv = cand_val + (size_t)row * C;
      const int* ci = cand_idx + (size_t)row * C;
      for (int i = lane; i < C; i += 32) {
        const int id = ci[i];
        const float v = cv[i];
        sidx[i] = id;
        skey[i] = (id >= 0 && v > 0.0f) ? __float_as_uint(v) : 0u;  // only positive candidates compete
      }
      __syncwarp();
      // threshold: the largest t with count(key >= t) >= k (0 when fewer than k candidates are positive)
      uint32_t t = 0;
      for (int bit = 30; bit >= 0; --bit) {
        const uint32_t trial = t | (1u << bit);
        int c = 0;
        for (int i = lane; i < C; i += 32) c += skey[i] >= trial;
        if (__reduce_add_sync(0xffffffffu, c) >= k) t = trial;
      }
      int above = 0;
      for (int i = lane; i < C; i += 32) above += skey[i] > t;
      above = __reduce_add_sync(0xffffffffu, above);
      const int ties_wanted = (t == 0u) ? 0 : k - above;  // t == 0: every positive candidate is in, nothing equals t
      // compaction of the winners in slot order
      int n_win = 0, ties_seen = 0;
      for (int base = 0; base < C; base += 32) {
        const int i = base + lane;
        const uint32_t key = i < C ? skey[i] : 0u;
        const bool eq = t != 0u && key == t;
        const unsigned eq_ballot = __ballot_sync(0xffffffffu, eq);
        const bool win = key > t || (eq && ties_seen + __popc(eq_ballot & lt_mask) < ties_wanted);
        const unsigned win_ballot = __ballot_sync(0xffffffffu, win);
        if (win) {
          const int pos = n_win + __popc(win_ballot & lt_mask);
          wkey[pos] = key;
          wslot[pos] = i;
        }
        n_win += __popc(win_ballot);
        ties_seen += __popc(eq_ballot);
      }
      __syncwarp();
      // place of each of this shard's winners among this shard's winners (value descending, earlier slot first
      // among equals)
      for (int w = lane; w < n_win; w += 32) {
        const int slot = wslot[w];
        if (slot < own_lo || slot >= own_hi) continue;
        const uint32_t key = wkey[w];
        int place = 0;
        for (int j = 0; j < n_win; ++j) {
          const uint32_t u = wkey[j];
          const int sj = wslot[j];
          place += (sj >= own_lo && sj < own_hi) && ((u > key) || (u == key && sj < slot));
        }
        const int id = sidx[slot];
        const float v = __uint_as_float(key);
        oidx[place] = id;
        oval[place] = (!emit_gated && gate != nullptr) ? v / gate[id] : v;
      }
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
  const size_t smem = (size_t)MERGE_WARPS * (2 * (size_t)C + 4 * (size_t)k) * 4;
  if (smem > 200 * 1024) return (int)cudaErrorInvalidValue;
  if (comm.mode != kMergePush && (out_idx == nullptr || out_val == nullptr)) return (int)cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(topk_merge_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  int blocks = (M + MERGE_WARPS - 1) / MERGE_WARPS;
  if (blocks > 148 * 8) blocks = 148 * 8;
  topk_merge_kernel<<<blocks, MERGE_WARPS * 32, smem, stream>>>(cand_val, cand_idx, M, C, k, gate, own_lo, own_hi,
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
constexpr int RT_BOUND_K = RT_THREADS * RT_MAXIMA / 2;  // (about 1.4 k candidates there, k + a few for small k)

__device__ __forceinline__ float gated_value(const __nv_bfloat16* __restrict__ hrow, const float* __restrict__ gate,
                                             const uint8_t* __restrict__ alive, int c) {
  float v = __bfloat162float(hrow[c]);
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
__device__ __noinline__ void row_topk_radix(const __nv_bfloat16* __restrict__ hrow, int row, int N, int k, const float* __restrict__ gate,
                                            const uint8_t* __restrict__ alive, int* __restrict__ out_idx, float* __restrict__ out_val) {
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
  for (int i = threadIdx.x; i < k; i += RT_THREADS) {
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
        out_idx[(size_t)row * k + pos] = c;
        out_val[(size_t)row * k + pos] = (gate != nullptr) ? v / gate[c] : v;
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

__global__ void __launch_bounds__(RT_THREADS, 5)
row_topk_kernel(const __nv_bfloat16* __restrict__ H, long long ldh, int M, int N, int k,
                const float* __restrict__ gate, const uint8_t* __restrict__ alive, int vec, int* __restrict__ out_idx,
                float* __restrict__ out_val) {
  const int row = blockIdx.x;
  if (row >= M) return;
  const __nv_bfloat16* hrow = H + (long long)row * ldh;
  __shared__ unsigned s_bits[RT_CAP];
  __shared__ int s_col[RT_CAP];
  __shared__ unsigned s_count[2][RT_WARPS];
  __shared__ int s_n, s_cursor;
  bool use_radix = k > RT_BOUND_K;
  if (!use_radix) {
    if (threadIdx.x == 0) { s_n = 0; s_cursor = 0; }
    // ---- pass 1: maxima of this thread's eight column groups (non-positive values and NaN never enter)
    float mx[RT_MAXIMA];
#pragma unroll
    for (int i = 0; i < RT_MAXIMA; ++i) mx[i] = 0.0f;
#pragma unroll 4
    for (int c = threadIdx.x * 8; c < N; c += RT_THREADS * 8) {
      float v[8];
      gated_values8(hrow, gate, alive, c, N, vec != 0, v);
#pragma unroll
      for (int i = 0; i < 8; ++i) mx[i] = fmaxf(mx[i], v[i]);
    }
    __syncthreads();
    unsigned mb[RT_MAXIMA];
#pragma unroll
    for (int i = 0; i < RT_MAXIMA; ++i) mb[i] = __float_as_uint(mx[i]);
    const unsigned bound = descend(mb, k, 16, s_count);
    // ---- pass 2: columns at or above the bound
#pragma unroll 2
    for (int c = threadIdx.x * 8; c < N; c += RT_THREADS * 8) {
      float v[8];
      gated_values8(hrow, gate, alive, c, N, vec != 0, v);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const unsigned b = __float_as_uint(v[i]);
        if (v[i] > 0.0f && b >= bound) {
          const int pos = atomicAdd(&s_n, 1);
          if (pos < RT_CAP) { s_bits[pos] = b; s_col[pos] = c + i; }
        }
      }
    }
    __syncthreads();
    const int n_cand = s_n;
    use_radix = n_cand > RT_CAP;  // (uniform)
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
          out_idx[(size_t)row * k + pos] = c;
          out_val[(size_t)row * k + pos] = gate != nullptr ? v / gate[c] : v;
        }
      };
      for (int j = threadIdx.x; j < n_cand; j += RT_THREADS)
        if (s_bits[j] > thr) place(j);
      __syncthreads();
      for (int j = threadIdx.x; j < n_cand; j += RT_THREADS)
        if (s_bits[j] == thr) place(j);
      for (int j = n_cand + threadIdx.x; j < k; j += RT_THREADS) {
        out_idx[(size_t)row * k + j] = -1;
        out_val[(size_t)row * k + j] = 0.0f;
      }
      return;
    }
  }
  row_topk_radix(hrow, row, N, k, gate, alive, out_idx, out_val);
}

int row_topk_launch(const __nv_bfloat16* H, long long ldh, int M, int N, int k, const float* gate,
                    const uint8_t* alive, int* out_idx, float* out_val, cudaStream_t stream) {
  const bool vec = N % 8 == 0 && ldh % 8 == 0 && reinterpret_cast<uintptr_t>(H) % 16 == 0 && reinterpret_cast<uintptr_t>(gate) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(alive) % 8 == 0;
  row_topk_kernel<<<M, RT_THREADS, 0, stream>>>(H, ldh, M, N, k, gate, alive, vec ? 1 : 0, out_idx, out_val);
  return (int)cudaGetLastError();
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
// ESTIMATE: h is only an estimate of x . W^T (fp32_gemm.cu). What is selected, and the selected values, are those of the fp32 sum in
// ascending order of k with one rounding per term. That sum lies within e = rel * xn * wn of the estimate, xn and wn the 2-norms of the
// row of x and the row of W (Cauchy-Schwarz bounds the sum of the magnitudes of the terms by their product; rel: see estimate_rel).
// Bias, norm and rounding are monotone, so the same operations on h - e and h + e, with the norm rounded down and up, enclose a positive g.
// The k-th largest lower end of the group maxima is reached by at least k columns, and whatever is selected has its upper end at or
// above it: those columns are summed up in order before the exact selection. Norms and wn come as two bf16 in one word: what bounds
// this kernel is the columns' arrays out of the L2 cache, twice for every row (4096 x 24576 x 768, k 50: 554 us with both in fp32, 506 so; a margin of 2^-8 of the bound, which the error could exceed,
// took 508). Rows with fewer than k positive values cost no more than others (1.16 ms for product and selection, 77 ms when such
// rows were summed up in order as a whole), and with every row listed it is 6.5 ms at 4096 x 32768 x 2048 (torch operations: 12.6).
// Columns that the bound says nothing about (wn is infinite there) are among them; rows with more such columns than there is room for are listed, multiplied in order as a whole
// (rows_product.cu) and selected from exactly. All decisions are taken on the device.
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned topk_key(float g) {
  const unsigned b = __float_as_uint(g);
  if ((b & 0x7fffffffu) > 0x7f800000u || b == 0xff800000u) return 0x7fffffffu;
  return (int)b > 0 ? b : 0u;
}
// (the intrinsics flush subnormals under this build's flags)
#define LMSAE_F32_OP(name, op)                                             \
  __device__ __forceinline__ float name(float a, float b) {                \
    float r;                                                               \
    asm(op " %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));                     \
    return r;                                                              \
  }
LMSAE_F32_OP(add_rn, "add.rn.f32")
LMSAE_F32_OP(mul_rn, "mul.rn.f32")
LMSAE_F32_OP(mul_up, "mul.rp.f32")
LMSAE_F32_OP(div_rn, "div.rn.f32")
#undef LMSAE_F32_OP
__device__ __forceinline__ float fma_rn(float a, float b, float c) {
  float r;
  asm("fma.rn.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ bool below(float a, float b) {  // a < b: false for a NaN, subnormals as they are
  int r;
  asm("{\n\t.reg .pred p;\n\tsetp.lt.f32 p, %1, %2;\n\tselp.s32 %0, 1, 0, p;\n\t}" : "=r"(r) : "f"(a), "f"(b));
  return r != 0;
}
__device__ __forceinline__ bool not_finite(float x) { return (__float_as_uint(x) & 0x7fffffffu) >= 0x7f800000u; }

// rel for sums of K terms, in units of 2^-24 (what the parts add up to):
//   K        roundings of the sum in order, one per term
//   K / 128  roundings of the estimate's slices added up
//   384      accumulations within a slice of 128 terms: the last eight instructions add sixteen full-size products each to what is there,
//            and each of these 17 operands may lose a unit to the alignment (136); the 40 before them add parts of 2^-8 and less (3);
//            the rest is margin for what the hardware does not document (measured: 2 units in all)
//   16       the three products that are left out (2^-25), the rounding of the ends themselves (|h| is at most about xn wn), and room
// The norms are rounded up by 5 % where they are made, which covers their own rounding and K 2^-24 << 1.
__host__ __device__ __forceinline__ float estimate_rel(int K) { return ((float)K * 1.01f + 400.0f) * 5.9604645e-8f; }

struct TopkDenseParams {
  float* h;
  const float* x;  // ESTIMATE: [B, K] and [N, K], and what the split of x and of W left (fp32_gemm.cu)
  const float* W;
  const float* xn;
  const uint32_t* ends;
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
// ESTIMATE: an end of g, the lower one for rx with a sign and the lower words of `ends`, else the upper one; the norms as those words have them
template <bool ESTIMATE>
__device__ __forceinline__ void topk_dense_load(const TopkDenseParams& p, const float* __restrict__ h, int c, float rx, float (&g)[4], float (&n)[4]) {
  float b[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  uint32_t w[4] = {0x3f800000u, 0x3f800000u, 0x3f800000u, 0x3f800000u};  // norm 1, and in a word of `ends` also a 2-norm of 0
  const uint32_t* words = ESTIMATE ? p.ends + ((int)__float_as_uint(rx) < 0 ? 0 : p.N) : reinterpret_cast<const uint32_t*>(p.norm);
  if (p.vec) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(h + c));
    g[0] = a.x; g[1] = a.y; g[2] = a.z; g[3] = a.w;
    if (p.bias != nullptr) {
      const float4 t = __ldg(reinterpret_cast<const float4*>(p.bias + c));
      b[0] = t.x; b[1] = t.y; b[2] = t.z; b[3] = t.w;
    }
    if (words != nullptr) {
      const uint4 t = __ldg(reinterpret_cast<const uint4*>(words + c));
      w[0] = t.x; w[1] = t.y; w[2] = t.z; w[3] = t.w;
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const bool in = c + i < p.N;
      g[i] = in ? __ldg(h + c + i) : 0.0f;
      if (in && p.bias != nullptr) b[i] = p.bias[c + i];
      if (in && words != nullptr) w[i] = __ldg(words + c + i);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    n[i] = __uint_as_float(ESTIMATE ? w[i] & 0xffff0000u : w[i]);
    if constexpr (ESTIMATE) g[i] = fma_rn(rx, __uint_as_float(w[i] << 16), g[i]);
    if (p.bias != nullptr) g[i] = add_rn(g[i], b[i]);
    if (ESTIMATE || p.norm != nullptr) g[i] = mul_rn(g[i], n[i]);
  }
}

// x . w, fp32, in ascending order (K % 4 == 0)
__device__ __forceinline__ float dot_in_order(const float* __restrict__ x, const float* __restrict__ w, int K) {
  float s = 0.0f;
#pragma unroll 8
  for (int i = 0; i < K; i += 4) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(x + i)), b = __ldg(reinterpret_cast<const float4*>(w + i));
    s = fma_rn(a.x, b.x, s);
    s = fma_rn(a.y, b.y, s);
    s = fma_rn(a.z, b.z, s);
    s = fma_rn(a.w, b.w, s);
  }
  return s;
}

// Sum over the CTA, the same in every thread.
__device__ __forceinline__ int cta_count(int mine, unsigned (&words)[RT_WARPS]) {
  const unsigned total = __reduce_add_sync(0xffffffffu, (unsigned)mine);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) words[threadIdx.x >> 5] = total;
  __syncthreads();
  return (int)__reduce_add_sync(0xffffffffu, (threadIdx.x & 31) < RT_WARPS ? words[threadIdx.x & 31] : 0u);
}

template <bool ESTIMATE>
__device__ __forceinline__ void topk_dense_row(const TopkDenseParams& p, int row) {
  __shared__ unsigned s_key[RT_CAP];
  __shared__ int s_col[RT_CAP];
  __shared__ unsigned s_count[2][RT_WARPS];
  __shared__ int s_n, s_above, s_equal;
  const float* h = p.h + (size_t)row * p.N;
  float* out = p.out + (size_t)row * p.N;
  const int N = p.N, k = p.k;
  const float rx = ESTIMATE ? mul_up(estimate_rel(p.K), p.xn[row]) : 0.0f, rx_lo = __uint_as_float(__float_as_uint(rx) | 0x80000000u);
  if (threadIdx.x == 0) { s_n = 0; s_above = 0; s_equal = 0; }
  unsigned mx[RT_MAXIMA];
#pragma unroll
  for (int i = 0; i < RT_MAXIMA; ++i) mx[i] = 0u;
#pragma unroll 2
  for (int c = threadIdx.x * 8; c < N; c += RT_THREADS * 8) {
#pragma unroll
    for (int half = 0; half < 8; half += 4) {
      if (c + half >= N) break;
      float g[4], nm[4];
      topk_dense_load<ESTIMATE>(p, h, c + half, rx_lo, g, nm);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        // (ESTIMATE: where wn is infinite the lower end is -inf or NaN, and neither enters)
        if constexpr (ESTIMATE) mx[half + i] = __float_as_uint(fmaxf(__uint_as_float(mx[half + i]), g[i]));
        else mx[half + i] = max(mx[half + i], topk_key(g[i]));
      }
    }
  }
  unsigned thr = descend(mx, k, 16, s_count);  // a bound until the exact value is known (0: fewer than k positive maxima)
  const float nan = __uint_as_float(0x7fffffffu), thr_f = __uint_as_float(max(thr, 1u));
#pragma unroll 2
  for (int c = threadIdx.x * 8; c < N; c += RT_THREADS * 8) {
#pragma unroll
    for (int half = 0; half < 8; half += 4) {
      if (c + half >= N) break;
      float g[4], nm[4];
      topk_dense_load<ESTIMATE>(p, h, c + half, rx, g, nm);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const unsigned nb = __float_as_uint(nm[i]) & 0x7fffffffu;
        unsigned key = 0u;
        bool enters, bad = nb == 0u || nb > 0x7f800000u;
        if constexpr (ESTIMATE) {  // (where wn is infinite the upper end is +inf or NaN, and enters; its value is looked at below)
          enters = !below(g[i], thr_f);
        } else {
          key = topk_key(g[i]);
          enters = key != 0u && key >= thr;
          bad |= not_finite(g[i]);
        }
        if (enters) {
          const int pos = atomicAdd(&s_n, 1);
          if (pos < RT_CAP) { s_key[pos] = key; s_col[pos] = c + half + i; }
        }
        g[i] = bad ? nan : 0.0f;
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
  __syncthreads();  // (also: the zeros are written before what is written over them)
  const int n = s_n;
  if constexpr (ESTIMATE) {
    if (n > RT_CAP) {
      if (threadIdx.x == 0) p.todo[1 + atomicAdd(p.todo, 1)] = row;
      return;
    }
    const float* x = p.x + (size_t)row * p.K;
    // (neighbouring candidates to different warps: a few dozen of them in one or two warps wait for their rows of W alone, 536 us)
    for (int j = (threadIdx.x & 31) * RT_WARPS + (threadIdx.x >> 5); j < n; j += RT_THREADS) {
      const int c = s_col[j];
      float g = dot_in_order(x, p.W + (size_t)c * p.K, p.K);
      if (p.bias != nullptr) g = add_rn(g, p.bias[c]);
      unsigned nb = 1u;
      if (p.norm != nullptr) {
        g = mul_rn(g, p.norm[c]);
        nb = __float_as_uint(p.norm[c]) & 0x7fffffffu;
      }
      s_key[j] = topk_key(g);
      if (not_finite(g) || nb == 0u || nb > 0x7f800000u) out[c] = nan;  // (the last two are NaN already)
    }
    __syncthreads();
  }
  auto put = [&](int c, unsigned key) {
    if (key == 0x7fffffffu) return;  // (what is NaN already stays so)
    float v = __uint_as_float(key);
    if (p.norm != nullptr) v = div_rn(v, p.norm[c]);
    out[c] = v;
  };
  if (n <= RT_CAP) {
    if (n > k) {
      unsigned mine[RT_CAP / RT_THREADS];
#pragma unroll
      for (int i = 0; i < RT_CAP / RT_THREADS; ++i) {
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
        topk_dense_load<false>(p, h, c, 0.0f, g, nm);
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

template <bool ESTIMATE>
__global__ void __launch_bounds__(RT_THREADS, 5)
topk_dense_kernel(const TopkDenseParams p) {
  topk_dense_row<ESTIMATE>(p, blockIdx.x);
}

__global__ void __launch_bounds__(RT_THREADS, 5)
topk_dense_rows_kernel(const TopkDenseParams p) {
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
  p.h = const_cast<float*>(h); p.bias = bias; p.norm = norm; p.out = out; p.N = N; p.k = k;
  p.vec = N % 4 == 0 && ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(norm) |
                          reinterpret_cast<uintptr_t>(out)) % 16 == 0);
  topk_dense_kernel<false><<<B, RT_THREADS, 0, stream>>>(p);
  return (int)cudaGetLastError();
}

// The same with h an estimate of x W^T (and overwritten where it is too coarse). todo: int [1 + B], todo[0] zeroed.
int topk_estimate_launch(float* h, const float* x, const float* W, const float* xn, const uint32_t* ends, int K, const float* bias, const float* norm,
                         int B, int N, int k, int* todo, float* out, cudaStream_t stream) {
  if (B <= 0 || N <= 0) return 0;
  if (k < 1 || k > RT_BOUND_K || K < 1 || K > kEstimateMaxK || K % 4 != 0 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(W)) & 15) != 0)
    return (int)cudaErrorInvalidValue;
  TopkDenseParams p = {};
  p.h = h; p.x = x; p.W = W; p.xn = xn; p.ends = ends; p.K = K; p.todo = todo; p.bias = bias; p.norm = norm; p.out = out; p.N = N; p.k = k;
  p.vec = N % 4 == 0 && ((reinterpret_cast<uintptr_t>(h) | reinterpret_cast<uintptr_t>(bias) | reinterpret_cast<uintptr_t>(norm) |
                          reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(ends)) % 16 == 0);
  topk_dense_kernel<true><<<B, RT_THREADS, 0, stream>>>(p);
  RowsProductParams r = {};
  r.A = x; r.B = W; r.C = h; r.N = N; r.K = K; r.rows = todo; r.max_rows = B;
  const int e = rows_product_launch(r, false, stream);
  if (e != 0) return e;
  p.rows = todo;
  topk_dense_rows_kernel<<<B < 148 * 5 ? B : 148 * 5, RT_THREADS, 0, stream>>>(p);
  return (int)cudaGetLastError();
}

}  // namespace lmsae
