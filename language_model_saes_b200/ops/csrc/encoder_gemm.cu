// Encoder GEMM for sparse dictionaries on sm_100a:
//
//     H[m, n] = sum_k X[m, k] * W[n, k] + bias[n]          (X, W bf16 K-major; fp32 accumulate)
//
// with two optional epilogues that run while the next tile's MMAs are in flight:
//   * WRITE_H : store H as bf16 (the "hidden_pre" tensor of the reference encoder,
//               models/sae.py:323-331 in the reference project); with a gate and no top-k, H * gate[n] is stored;
//   * TOPK    : keep, per row, the k largest *gated* values g = H * gate[n] (gate = decoder row norm when
//               sparsity_include_decoder_norm is set, models/sae.py:333-341) that are > 0, without ever
//               writing the dense pre-activation matrix. Each CTA sweeps a contiguous range of N-tiles for
//               one 128-row panel, so the running top-k state lives in shared memory for the whole sweep;
//               at the end it emits k (value, column) candidates per row for its range. A small merge
//               kernel (topk_merge.cu) combines the ranges (and, under feature sharding, the ranks).
//
// Structure (one CTA per SM, 256 threads, 384 without top-k):
//   warp 0    : TMA producer (one elected lane) -> STAGES-deep ring of {A 128x64, B 256x64} bf16 tiles,
//               128-byte swizzle, no cluster multicast
//   warp 1    : tcgen05.mma issuer (one elected lane), UMMA 128x256x16, accumulators in TMEM,
//               two 256-column accumulator buffers so the epilogue of tile i overlaps the MMAs of tile i+1
//   warp 2    : TMEM allocation / release
//   warps 4-7 : epilogue; thread r of the warpgroup owns accumulator row r (TMEM lane r); without top-k warps 8-11 take half of its columns
// Every mbarrier wait is bounded; on expiry the CTA records a status code, raises a CTA-wide abort flag,
// drains and frees its TMEM.
//
// PAIR variant (tcgen05 cta_group::2): two CTAs on neighbouring SMs form a cluster and work on two adjacent
// 128-row panels with ONE 256x256x16 instruction stream issued by the leader (cluster rank 0). Each CTA loads
// its own A tile and only HALF of the B tile (128 of the 256 dictionary rows), so a stage is 32 KB instead of
// 48 KB per CTA: B crosses L2 -> shared memory once per pair, and the ring is 4-5 stages deep even with the
// top-k candidate buffers resident. Both producers complete their bytes on the LEADER's "full" barrier; the
// leader's commits arrive on the "empty" / "accumulator full" barriers of BOTH CTAs; both epilogues release an
// accumulator buffer on the leader's "accumulator empty" barrier. Each CTA's epilogue is unchanged: it reads
// its own 128 TMEM lanes (its panel's rows) x 256 columns.
#include "common.cuh"
#include "kernels.h"

namespace lmsae {

constexpr int BM = 128;
constexpr int BN = 256;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int A_STAGE_BYTES = BM * BK * 2;  // 16 KB
constexpr int TMEM_COLS = 512;
// Epilogue warps: four with the top-k (a thread keeps a row's buffer), else eight, two per accumulator row with half of the columns each:
// a single warp per scheduler waits for every TMEM load. H of 4096 x 24576 x 768: 135 -> 126 us.
__host__ __device__ constexpr int epilogue_warps(bool topk) { return topk ? 4 : 8; }

// Entries of a row's candidate buffer (CAP): the k best so far plus room for what is appended until the next selection. A step of
// the sweep appends at most 16, so k + 16 entries suffice; more room means fewer selections, but costs ring stages.
// NARROW buffers hold columns as 16-bit offsets from the start of the range (codes from kCarried on: entry code - kCarried of the
// resumed state). 4096 rows x 24576 columns, K 768, k 50 / 64: 204 / 322 us with 80 entries and five stages, 191 / 207 with 128
// and four; k 32: 173 and 177. But K 4096 x 131072 columns is bound by the tensor cores and takes 5 % longer with four stages than with five.
constexpr int kNarrowTiles = 255;
constexpr int kCarried = kNarrowTiles * BN;

template <int STAGES, int CAP, bool PAIR, bool NARROW, bool F32>
struct SmemLayout {
  static constexpr int kBRows = PAIR ? BN / 2 : BN;       // dictionary rows of a B tile held by one CTA
  static constexpr int kBStageBytes = kBRows * BK * 2;    // 16 KB (pair) / 32 KB
  static constexpr int kStageBytes = A_STAGE_BYTES + kBStageBytes;
  static constexpr int kStageOff = 0;
  static constexpr int kSlotValOff = STAGES * kStageBytes;
  static constexpr int kSlotIdxOff = kSlotValOff + BM * CAP * 4;
  static constexpr int kColOff = kSlotIdxOff + BM * CAP * (NARROW ? 2 : 4);   // per epilogue warp: bias and gate of the 32 columns at work
  static constexpr int kEpilogueWarps = epilogue_warps(CAP != 0);
  static constexpr int kStoreOff = kColOff + kEpilogueWarps * 64 * 4;  // per epilogue warp: 32 x 32 values on their way to whole sectors of H (no top-k)
  static constexpr int kMaxOff = kStoreOff + (CAP == 0 ? kEpilogueWarps * (F32 ? 4096 : 2048) : 0);  // per 32 rows: maxima of a tile's eight groups of columns, [8][32 rows]
  static constexpr int kBarOff = kMaxOff + (CAP == 0 ? 4 * 1024 : 0);
  static constexpr int kNumBars = 2 * STAGES + 4;
  static constexpr int kTmemPtrOff = kBarOff + kNumBars * 8;
  static constexpr int kAbortOff = kTmemPtrOff + 4;
  static constexpr int kTotal = kAbortOff + 4;
  static constexpr int kDynamicBytes = kTotal + 1024;  // slack for manual 1024-byte alignment
};

struct RowState {
  int n;      // entries in the row's buffer
  float tau;  // at least k of them are >= tau: a column has to beat it
};

// Element-wise over pairs in one instruction each.
__device__ __forceinline__ void add_pair(float& a0, float& a1, float b0, float b1) {
  asm("{\n\t.reg .b64 ra, rb;\n\tmov.b64 ra, {%0, %1};\n\tmov.b64 rb, {%2, %3};\n\tadd.rn.f32x2 ra, ra, rb;\n\tmov.b64 {%0, %1}, ra;\n\t}"
      : "+f"(a0), "+f"(a1)
      : "f"(b0), "f"(b1));
}
__device__ __forceinline__ void mul_pair(float& a0, float& a1, float b0, float b1) {
  asm("{\n\t.reg .b64 ra, rb;\n\tmov.b64 ra, {%0, %1};\n\tmov.b64 rb, {%2, %3};\n\tmul.rn.f32x2 ra, ra, rb;\n\tmov.b64 {%0, %1}, ra;\n\t}"
      : "+f"(a0), "+f"(a1)
      : "f"(b0), "f"(b1));
}

// The larger one, NaN where one is NaN.
__device__ __forceinline__ float max_nan(float a, float b) {
  float r;
  asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// Entry {value, column} to shared memory where the condition holds: predicated, because a branch per column costs more than the
// rest of the epilogue (one warp per scheduler). The address of the next entry is a NEW register of the caller's: advanced in
// place, it would have to wait for every store to have read it (23 cycles a column).
template <bool NARROW>
__device__ __forceinline__ void store_entry_if(bool cond, uint32_t val_addr, uint32_t col_addr, uint32_t bits, uint32_t col) {
  if constexpr (NARROW)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.b32 [%1], %3;\n\t@p st.shared.b16 [%2], %4;\n\t}" ::"r"((uint32_t)cond),
                 "r"(val_addr), "r"(col_addr), "r"(bits), "h"((unsigned short)col)
                 : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.b32 [%1], %3;\n\t@p st.shared.b32 [%2], %4;\n\t}" ::"r"((uint32_t)cond),
                 "r"(val_addr), "r"(col_addr), "r"(bits), "r"(col)
                 : "memory");
}

// A row's buffer: entry s has its value at [s][row] of one array and its column at [s][row] of the other, both BM rows wide.
template <int CAP, bool NARROW>
struct RowBuffer {
  uint32_t val;       // shared-memory address of entry 0's value
  uint32_t val0, col0;  // the two arrays
  __device__ __forceinline__ uint32_t col_of(uint32_t val_addr) const {
    return NARROW ? ((val_addr - val0) >> 1) + col0 : val_addr - val0 + col0;
  }
  __device__ __forceinline__ uint32_t value(int s) const {
    uint32_t x;
    asm volatile("ld.shared.b32 %0, [%1];" : "=r"(x) : "r"(val + s * (BM * 4)) : "memory");
    return x;
  }
  __device__ __forceinline__ uint32_t column(int s) const {
    const uint32_t a = col_of(val + s * (BM * 4));
    if constexpr (NARROW) {
      unsigned short x;
      asm volatile("ld.shared.b16 %0, [%1];" : "=h"(x) : "r"(a) : "memory");
      return x;
    } else {
      uint32_t x;
      asm volatile("ld.shared.b32 %0, [%1];" : "=r"(x) : "r"(a) : "memory");
      return x;
    }
  }
};

// Cuts the buffers of a warp's 32 rows (one per lane) down to at most `limit` >= k entries each without losing any of the k
// largest: a bisection (of values first, then of their bit patterns, which order positive floats) for a bound that between k and
// `limit` entries reach. Where equal values leave no such bound, the first of them fill up to k. Rows that hold no more than
// `limit` entries stay as they are. Order is kept.
template <int CAP, bool NARROW>
__device__ __noinline__ RowState select_entries(RowBuffer<CAP, NARROW> buf, RowState st, int k, int limit) {
  uint32_t w[CAP];
  uint32_t top[4] = {0u, 0u, 0u, 0u};  // (four chains at a time: a single one is bound by the latency of its links)
#pragma unroll
  for (int s = 0; s < CAP; ++s) w[s] = buf.value(s);
#pragma unroll
  for (int s = 0; s < CAP; ++s) {
    w[s] = s < st.n ? w[s] : 0u;
    top[s & 3] = max(top[s & 3], w[s]);
  }
  const bool mine = st.n > limit;
  bool active = mine;
  uint32_t lo = max(__float_as_uint(st.tau), 1u), hi = max(max(top[0], top[1]), max(top[2], top[3])) + 1u;  // count(>= lo) >= k > count(>= hi)
  int at_lo = st.n;
  for (int step = 0; __any_sync(0xffffffffu, active); ++step) {
    uint32_t mid = step < 8 ? __float_as_uint(0.5f * __uint_as_float(lo) + 0.5f * __uint_as_float(hi - 1u)) : lo + ((hi - lo) >> 1);
    mid = min(max(mid, lo + 1u), hi - 1u);
    int c[4] = {0, 0, 0, 0};
#pragma unroll
    for (int s = 0; s < CAP; ++s) c[s & 3] += w[s] >= mid;
    if (active) {
      const int n = (c[0] + c[1]) + (c[2] + c[3]);
      if (n >= k) { lo = mid; at_lo = n; } else { hi = mid; }
      active = at_lo > limit && hi - lo > 1u;
    }
  }
  const bool tied = mine && at_lo > limit;  // too many entries equal to the bound
  uint32_t at = buf.val;
  if (!__any_sync(0xffffffffu, tied)) {
    const uint32_t bound = mine ? lo : 0xffffffffu;
#pragma unroll
    for (int b = 0; b < CAP; b += 16) {
      uint32_t id[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) id[i] = buf.column(b + i);  // (read before anything at or behind them is overwritten)
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const bool keep = w[b + i] >= bound;
        store_entry_if<NARROW>(keep, at, buf.col_of(at), w[b + i], id[i]);
        at = at + (keep ? BM * 4 : 0);
      }
    }
  } else {
    int ties = tied ? k : CAP;
    if (tied) {
#pragma unroll
      for (int s = 0; s < CAP; ++s) ties -= w[s] > lo;
    }
#pragma unroll
    for (int s = 0; s < CAP; ++s) {
      const uint32_t id = buf.column(s);
      const bool tie = w[s] == lo, keep = mine && (w[s] > lo || (tie && ties > 0));
      ties -= tie;
      store_entry_if<NARROW>(keep, at, buf.col_of(at), w[s], id);
      at = at + (keep ? BM * 4 : 0);
    }
  }
  if (mine) {
    st.n = (int)((at - buf.val) / (BM * 4));
    st.tau = __uint_as_float(lo);
  }
  return st;
}

// F32: H is stored in fp32 (without top-k).
template <bool WRITE_H, bool TOPK, int STAGES, int KS, int CAP, bool PAIR, bool NARROW, bool F32>
__global__ void __launch_bounds__(128 + 32 * epilogue_warps(TOPK), 1)
enc_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                const EncGemmParams p) {
  pdl_wait();
  using L = SmemLayout<STAGES, CAP, PAIR, NARROW, F32>;
  constexpr int STAGE_BYTES = L::kStageBytes;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));

  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tmem_full_bar = empty_bar + STAGES;
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem + L::kTmemPtrOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kAbortOff);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  // work unit = one CTA (one panel) or one CTA pair (two adjacent panels); units of a split are consecutive
  const uint32_t cta_rank = PAIR ? cluster_ctarank() : 0u;
  const bool leader = cta_rank == 0;
  const int unit = PAIR ? (int)(blockIdx.x >> 1) : (int)blockIdx.x;
  const int units_per_split = PAIR ? p.num_panels / 2 : p.num_panels;
  // ragged deal (p.units != 0): the first `extra` panel units get base + 1 column ranges, the others base; units of one
  // range index are consecutive within their group, so the CTAs that run together sweep the same B tiles
  int panel_unit, split, my_splits;
  if (p.units == 0) {
    panel_unit = unit % units_per_split;
    split = unit / units_per_split;
    my_splits = p.num_splits;
  } else {
    const int base = p.units / units_per_split, extra = p.units % units_per_split;
    const int first = extra * (base + 1);
    if (unit < first) {
      panel_unit = unit % extra;
      split = unit / extra;
      my_splits = base + 1;
    } else {
      const int rest = units_per_split - extra;
      panel_unit = extra + (unit - first) % rest;
      split = (unit - first) / rest;
      my_splits = base;
    }
  }
  const int panel = PAIR ? panel_unit * 2 + (int)cta_rank : panel_unit;
  const int num_n_tiles = (p.N + BN - 1) / BN;
  const int tile_begin = (int)(((long long)split * num_n_tiles) / my_splits);
  const int tile_end = (int)(((long long)(split + 1) * num_n_tiles) / my_splits);
  const int num_k_stages = (p.K + BK - 1) / BK;
  const int m0 = panel * BM;

  if (threadIdx.x == 0) {
    for (int i = 0; i < STAGES; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    mbar_init(&tmem_full_bar[0], 1);
    mbar_init(&tmem_full_bar[1], 1);
    for (int i = 0; i < 2; ++i) mbar_init(&tmem_empty_bar[i], epilogue_warps(TOPK) * (PAIR ? 2 : 1));  // epilogue warps of the CTA (of both CTAs of a pair)
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&tmap_b);
  }
  if (warp == 2) {
    if constexpr (PAIR) {
      tmem_alloc_pair(tmem_ptr_smem, TMEM_COLS);
      tmem_relinquish_pair();
    } else {
      tmem_alloc(tmem_ptr_smem, TMEM_COLS);
      tmem_relinquish();
    }
  }
  tc_fence_before();
  __syncthreads();
  if constexpr (PAIR) cluster_sync_all();  // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      const int k_stages_per_head = p.heads > 1 ? num_k_stages / p.heads : num_k_stages;
      for (int tile = tile_begin; tile < tile_end && ok; ++tile) {
        const int n0 = tile * BN;
        for (int ks = 0; ks < num_k_stages; ++ks, ++it) {
          const int s = it % STAGES;
          const uint32_t parity = ((it / STAGES) & 1) ^ 1;
          // head-summed encoders: K block ks belongs to head h and reads that head's rows of the weight map
          const int head = ks / k_stages_per_head;
          const int bk = (ks - head * k_stages_per_head) * BK;
          const int brow = n0 + head * p.b_rows_per_head;
          if (!mbar_wait_bounded(&empty_bar[s], parity, abort_flag)) {
            report_status(p.status, kTimeoutEmptyBarrier, (int)it);
            *abort_flag = 1;
            ok = false;
            break;
          }
          uint8_t* a_dst = smem + L::kStageOff + s * STAGE_BYTES;
          uint8_t* b_dst = a_dst + A_STAGE_BYTES;
          if constexpr (PAIR) {
            // the leader's barrier counts the bytes of both CTAs; bytes landing before the leader has
            // announced them only make the pending count negative for a moment
            if (leader) mbar_arrive_expect_tx(&full_bar[s], 2 * STAGE_BYTES);
            const uint32_t bar = mapa_u32(smem_u32(&full_bar[s]), 0);
            tma_load_2d_pair(a_dst, &tmap_a, bar, ks * BK, m0);
            tma_load_2d_pair(b_dst, &tmap_b, bar, bk, brow + (int)cta_rank * L::kBRows);
          } else {
            mbar_arrive_expect_tx(&full_bar[s], STAGE_BYTES);
            tma_load_2d(a_dst, &tmap_a, &full_bar[s], ks * BK, m0);
            tma_load_2d(b_dst, &tmap_b, &full_bar[s], bk, brow);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (pair: leader CTA only)
    if ((!PAIR || leader) && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(PAIR ? 2 * BM : BM, BN);
      uint32_t it = 0;
      bool ok = true;
      int lt = 0;
      for (int tile = tile_begin; tile < tile_end && ok; ++tile, ++lt) {
        const int buf = lt & 1;
        const uint32_t acc_parity = ((lt >> 1) & 1) ^ 1;
        if (!mbar_wait_bounded(&tmem_empty_bar[buf], acc_parity, abort_flag)) {
          report_status(p.status, kTimeoutTmemEmpty, lt);
          *abort_flag = 1;
          break;
        }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + (uint32_t)(buf * BN);
        for (int ks = 0; ks < num_k_stages; ++ks, ++it) {
          const int s = it % STAGES;
          const uint32_t parity = (it / STAGES) & 1;
          if (!mbar_wait_bounded(&full_bar[s], parity, abort_flag)) {
            report_status(p.status, kTimeoutFullBarrier, (int)it);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + L::kStageOff + s * STAGE_BYTES);
          const uint32_t b_addr = a_addr + A_STAGE_BYTES;
          const uint64_t a_desc = make_sw128_kmajor_desc(a_addr);
          const uint64_t b_desc = make_sw128_kmajor_desc(b_addr);
#pragma unroll
          for (int kk = 0; kk < BK / UMMA_K; ++kk) {
            // +32 bytes per 16-element K step: the start-address field is in 16-byte units
            const uint32_t acc = (ks > 0 || kk > 0) ? 1u : 0u;
            if constexpr (PAIR) {
              umma_bf16_ss_pair(tmem_d, a_desc + (uint64_t)(kk * 2), b_desc + (uint64_t)(kk * 2), idesc, acc);
            } else {
              umma_bf16_ss(tmem_d, a_desc + (uint64_t)(kk * 2), b_desc + (uint64_t)(kk * 2), idesc, acc);
            }
          }
          // stage reusable (in both CTAs of a pair) once these MMAs have read it
          if constexpr (PAIR) umma_commit_pair(&empty_bar[s], 3); else umma_commit(&empty_bar[s]);
        }
        if (ok) {
          if constexpr (PAIR) umma_commit_pair(&tmem_full_bar[buf], 3); else umma_commit(&tmem_full_bar[buf]);
        }
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ epilogue
    const int q = warp & 3;             // TMEM lane quarter of this warp
    const int part = (warp - 4) >> 2;   // and its share of the columns
    constexpr int CHUNKS = BN / 32 * 4 / epilogue_warps(TOPK);
    const int row_in_tile = q * 32 + lane;
    const int row = m0 + row_in_tile;
    const bool row_ok = row < p.M;
    // Running top-k of this thread's row: columns above tau are APPENDED to the row's buffer in shared memory (entry-major,
    // [CAP][128 rows]: no bank conflicts); when a row of the warp has no room left, all 32 are cut back and get a new tau at
    // once. An append is a few predicated instructions, and the number of selections grows with the logarithm of the
    // columns; replacing the smallest of k entries column by column took some 400 cycles for each of the several hundred
    // columns per row that enter, serialised over the lanes of a warp: 4096 x 24576 x 768, k 50: 332 -> 190 us.
    RowState st = {0, row_ok ? 0.0f : __int_as_float(0x7f800000)};
    RowBuffer<CAP, NARROW> rowbuf;
    rowbuf.val0 = smem_u32(smem + L::kSlotValOff);
    rowbuf.col0 = smem_u32(smem + L::kSlotIdxOff);
    rowbuf.val = rowbuf.val0 + row_in_tile * 4;
    const int col_base = NARROW ? p.n_index_offset + tile_begin * BN : 0;  // what the stored columns count from
    // Bias and gate of the columns at work come through shared memory, fetched one step ahead by a coalesced load per warp
    // (read per thread they were a miss in L1 for every step); columns past the end have gate 0.
    float* col_bias = reinterpret_cast<float*>(smem + L::kColOff) + (warp - 4) * 64;
    float* col_gate = col_bias + 32;
    const float* gate_src = !TOPK && p.gate == nullptr ? p.max_gate : p.gate;
    float* tile_max = reinterpret_cast<float*>(smem + L::kMaxOff) + q * 256 + lane;
    float next_bias = 0.0f, next_gate = 0.0f;
    auto fetch_columns = [&](int c) {
      const bool in = c + lane < p.N;
      next_bias = in && p.bias != nullptr ? __ldg(p.bias + c + lane) : 0.0f;
      next_gate = !in ? 0.0f : gate_src != nullptr ? __ldg(gate_src + c + lane) : 1.0f;
    };
    if constexpr (TOPK) {
      if (p.resume_topk && row_ok) {
        // continue the sweep of an earlier launch: its result for (row, this column range) is the state
        const long long o = (long long)row * ((long long)p.num_splits * KS) + (long long)split * KS;
        for (int s = 0; s < KS; ++s) {
          const int ix = p.cand_idx[o + s];
          if (ix < 0) continue;
          const uint32_t a = rowbuf.val + st.n * (BM * 4);
          store_entry_if<NARROW>(true, a, rowbuf.col_of(a), __float_as_uint(p.cand_val[o + s]), NARROW ? kCarried + s : ix);
          ++st.n;
        }
      }
      __syncwarp();
    }
    fetch_columns(tile_begin * BN + part * CHUNKS * 32);
    int lt = 0;
    bool ok = true;
    for (int tile = tile_begin; tile < tile_end && ok; ++tile, ++lt) {
      const int buf = lt & 1;
      const uint32_t parity = (lt >> 1) & 1;
      if (!__all_sync(0xffffffffu, mbar_wait_bounded(&tmem_full_bar[buf], parity, abort_flag))) {
        if (lane == 0) report_status(p.status, kTimeoutTmemFull, lt);
        *abort_flag = 1;
        ok = false;
        break;
      }
      tc_fence_after();
      const int n0 = tile * BN;
      const uint32_t taddr_row = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN);
      if constexpr (WRITE_H && !TOPK) {
        if (p.maxima != nullptr)
          for (int c = 0; c < CHUNKS; ++c) tile_max[(part * CHUNKS + c) * 32] = __int_as_float(0xff800000);  // (groups past the last column)
      }
#pragma unroll 1
      for (int chunk = part * CHUNKS; chunk < (part + 1) * CHUNKS; ++chunk) {
        const int c0 = n0 + chunk * 32;
        if (c0 >= p.N) break;  // uniform across the CTA
        __syncwarp();  // (the previous step's values have been read)
        col_bias[lane] = next_bias;
        col_gate[lane] = next_gate;
        __syncwarp();
        fetch_columns(chunk + 1 < (part + 1) * CHUNKS ? c0 + 32 : n0 + BN + part * CHUNKS * 32);
        uint32_t r[32];
        tmem_ld_32x32b_x32(taddr_row + (uint32_t)(chunk * 32), r);
        tmem_wait_ld();
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
#pragma unroll
        for (int j = 0; j < 32; j += 4) {
          const float4 b4 = *reinterpret_cast<const float4*>(col_bias + j);
          add_pair(v[j], v[j + 1], b4.x, b4.y);
          add_pair(v[j + 2], v[j + 3], b4.z, b4.w);
        }
        if constexpr (WRITE_H && TOPK) {  // (the ungated value)
          if (row_ok) {
            __nv_bfloat16* dst = p.H + (long long)row * p.ldh + c0;
#pragma unroll
            for (int j = 0; j < 32; j += 8)  // (N % 8 == 0)
              if (c0 + j < p.N)
                *reinterpret_cast<uint4*>(dst + j) = make_uint4(pack_bf16x2(v[j], v[j + 1]), pack_bf16x2(v[j + 2], v[j + 3]),
                                                                pack_bf16x2(v[j + 4], v[j + 5]), pack_bf16x2(v[j + 6], v[j + 7]));
          }
        }
        if (!F32 && (TOPK || p.gate != nullptr)) {
#pragma unroll
          for (int j = 0; j < 32; j += 4) {
            const float4 g4 = *reinterpret_cast<const float4*>(col_gate + j);
            mul_pair(v[j], v[j + 1], g4.x, g4.y);
            mul_pair(v[j + 2], v[j + 3], g4.z, g4.w);
          }
        }
        if constexpr (WRITE_H && !TOPK && F32) {
          // (as below, with 128 bytes of a row: eight lanes write a line)
          uint8_t* tile_s = smem + L::kStoreOff + (warp - 4) * 4096;
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<float4*>(tile_s + lane * 128 + ((j ^ (lane & 7)) * 16)) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
          if (p.maxima != nullptr) {
            float m[4] = {__int_as_float(0xff800000), __int_as_float(0xff800000), __int_as_float(0xff800000), __int_as_float(0xff800000)};
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              if (p.max_gate != nullptr) {
                const float4 g4 = *reinterpret_cast<const float4*>(col_gate + j);
                mul_pair(v[j], v[j + 1], g4.x, g4.y);
                mul_pair(v[j + 2], v[j + 3], g4.z, g4.w);
              }
#pragma unroll
              for (int i = 0; i < 4; ++i) m[i] = max_nan(m[i], v[j + i]);
            }
            tile_max[chunk * 32] = max_nan(max_nan(m[0], m[1]), max_nan(m[2], m[3]));
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int rr = i * 4 + (lane >> 3), j = lane & 7;
            const float4 o = *reinterpret_cast<const float4*>(tile_s + rr * 128 + ((j ^ (rr & 7)) * 16));
            if (m0 + q * 32 + rr < p.M && c0 + j * 4 < p.N)  // (N % 8 == 0)
              *reinterpret_cast<float4*>(p.H32 + (long long)(m0 + q * 32 + rr) * p.ldh + c0 + j * 4) = o;
          }
        }
        if constexpr (WRITE_H && !TOPK && !F32) {
          // A thread holds 64 bytes of its own row: through shared memory (16-byte pieces, swizzled: no bank conflicts), so that
          // four lanes write whole sectors of a row. Stored from the registers, every instruction touched 32 rows by half a
          // sector each: 4096 x 24576 x 768: 198 (with a gate: 425) -> 135 (149) us.
          uint8_t* tile_s = smem + L::kStoreOff + (warp - 4) * 2048;
          uint32_t w[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) w[j] = pack_bf16x2(v[2 * j], v[2 * j + 1]);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            *reinterpret_cast<uint4*>(tile_s + lane * 64 + ((j ^ ((lane >> 1) & 3)) * 16)) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
          if (p.maxima != nullptr) {  // of the values as they are stored
            float m[4] = {__int_as_float(0xff800000), __int_as_float(0xff800000), __int_as_float(0xff800000), __int_as_float(0xff800000)};
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const uint32_t w0 = w[j / 2], w1 = w[j / 2 + 1];
              float x0 = __uint_as_float(w0 << 16), x1 = __uint_as_float(w0 & 0xffff0000u), x2 = __uint_as_float(w1 << 16), x3 = __uint_as_float(w1 & 0xffff0000u);
              if (p.max_gate != nullptr) {
                const float4 g4 = *reinterpret_cast<const float4*>(col_gate + j);
                mul_pair(x0, x1, g4.x, g4.y);
                mul_pair(x2, x3, g4.z, g4.w);
              }
              m[0] = max_nan(m[0], x0); m[1] = max_nan(m[1], x1);
              m[2] = max_nan(m[2], x2); m[3] = max_nan(m[3], x3);
            }
            tile_max[chunk * 32] = max_nan(max_nan(m[0], m[1]), max_nan(m[2], m[3]));
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int rr = i * 8 + (lane >> 2), j = lane & 3;
            const uint4 o = *reinterpret_cast<const uint4*>(tile_s + rr * 64 + ((j ^ ((rr >> 1) & 3)) * 16));
            if (m0 + q * 32 + rr < p.M && c0 + j * 8 < p.N)  // (N % 8 == 0)
              *reinterpret_cast<uint4*>(p.H + (long long)(m0 + q * 32 + rr) * p.ldh + c0 + j * 8) = o;
          }
        }
        if constexpr (TOPK) {
#pragma unroll
          for (int h = 0; h < 32; h += 16) {
            float m[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) m[j] = fmaxf(fmaxf(v[h + j], v[h + 4 + j]), fmaxf(v[h + 8 + j], v[h + 12 + j]));
            const bool enters = fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3])) > st.tau;
            if (!__any_sync(0xffffffffu, enters)) continue;
            if (__any_sync(0xffffffffu, enters && st.n + 16 > CAP)) {
              int enter = 0;
#pragma unroll
              for (int j = 0; j < 16; ++j) enter += v[h + j] > st.tau;
              if (__any_sync(0xffffffffu, st.n + enter > CAP))
                st = select_entries<CAP, NARROW>(rowbuf, st, p.k, min(p.k + max(8, (CAP - p.k) / 4), CAP - 16));
            }
            uint32_t at = rowbuf.val + (uint32_t)st.n * (BM * 4);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const bool above = v[h + j] > st.tau;
              store_entry_if<NARROW>(above, at, rowbuf.col_of(at), __float_as_uint(v[h + j]), p.n_index_offset + c0 + h + j - col_base);
              at = at + (above ? BM * 4 : 0);
            }
            st.n = (int)((at - rowbuf.val) / (BM * 4));
          }
        }
      }
      if constexpr (WRITE_H && !TOPK) {
        if (p.maxima != nullptr && row_ok) {  // (a lane's own entries)
          const float* m = tile_max + part * CHUNKS * 32;
          static_assert(TOPK || CHUNKS == 4, "one store");
          *reinterpret_cast<float4*>(p.maxima + (long long)row * p.ld_maxima + tile * (BN / 32) + part * CHUNKS) = make_float4(m[0], m[32], m[64], m[96]);
        }
      }
      // release this accumulator buffer to the MMA warp
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        if constexpr (PAIR) mbar_arrive_cluster(mapa_u32(smem_u32(&tmem_empty_bar[buf]), 0));
        else mbar_arrive(&tmem_empty_bar[buf]);
      }
    }
    if constexpr (TOPK) {
      __syncwarp();
      st = select_entries<CAP, NARROW>(rowbuf, st, p.k, KS);
    }
    if constexpr (TOPK) if (ok && row_ok) {
      // emit this sweep's candidates (at least the k best, at most KS): [row][split * KS + slot]
      const long long o = (long long)row * ((long long)p.num_splits * KS) + (long long)split * KS;
      const bool whole = ((reinterpret_cast<uintptr_t>(p.cand_val) | reinterpret_cast<uintptr_t>(p.cand_idx)) & 15) == 0;  // (lists may be views)
      for (int s = 0; s < KS; s += 4) {
        float v[4];
        int ix[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const bool valid = s + i < st.n;
          v[i] = valid ? __uint_as_float(rowbuf.value(s + i)) : 0.0f;
          ix[i] = valid ? (int)rowbuf.column(s + i) : -1;
          // (an entry carried over from slot c sits at or before slot c: its column there is not overwritten yet)
          if (NARROW && valid) ix[i] = ix[i] >= kCarried ? p.cand_idx[o + ix[i] - kCarried] : ix[i] + col_base;
        }
        if (whole) {
          *reinterpret_cast<float4*>(p.cand_val + o + s) = make_float4(v[0], v[1], v[2], v[3]);
          *reinterpret_cast<int4*>(p.cand_idx + o + s) = make_int4(ix[0], ix[1], ix[2], ix[3]);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            p.cand_val[o + s + i] = v[i];
            p.cand_idx[o + s + i] = ix[i];
          }
        }
      }
      // a panel with fewer ranges than the lists have room for: its last range also marks the unused lists empty
      if (split == my_splits - 1) {
        for (int s = my_splits * KS; s < p.num_splits * KS; ++s) {
          const long long e = (long long)row * ((long long)p.num_splits * KS) + s;
          p.cand_val[e] = 0.0f;
          p.cand_idx[e] = -1;
        }
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) {
    // let copies that may still be in flight land before shared memory and TMEM go away
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    __syncthreads();
  }
  // pair: neither CTA may free TMEM or leave while the other can still touch its barriers, shared memory or
  // accumulator rows
  if constexpr (PAIR) cluster_sync_all();
  if (warp == 2) {
    tc_fence_after();
    if constexpr (PAIR) tmem_dealloc_pair(tmem_base, TMEM_COLS); else tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

// ---- host side -------------------------------------------------------------------------------
template <bool WRITE_H, bool TOPK, int STAGES, int KS, int CAP, bool PAIR, bool NARROW = false, bool F32 = false>
static cudaError_t launch_variant(const CUtensorMap& ta, const CUtensorMap& tb, const EncGemmParams& p,
                                  cudaStream_t stream) {
  using L = SmemLayout<STAGES, CAP, PAIR, NARROW, F32>;
  static_assert(L::kDynamicBytes <= 232448, "shared memory of one CTA exceeds 227 KB");
  auto kern = enc_gemm_kernel<WRITE_H, TOPK, STAGES, KS, CAP, PAIR, NARROW, F32>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynamicBytes);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.units != 0 ? p.units * (PAIR ? 2 : 1) : p.num_panels * p.num_splits);
  cfg.blockDim = dim3(128 + 32 * epilogue_warps(TOPK));
  cfg.dynamicSmemBytes = L::kDynamicBytes;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = PAIR ? 2 : 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  ++kernel_launches;
  return cudaLaunchKernelEx(&cfg, kern, ta, tb, p);
}

// mode: bit 0 = WRITE_H, bit 1 = TOPK, bit 2 = 3-stage ring for the plain single-CTA variant (a tuning probe),
// bit 3 = CTA-pair variant (needs an even number of panels; `tb` must then have a 128-row box),
// bit 4 = with bit 3 and TOPK: a shorter ring (under 200 KB of shared memory), which leaves room on the SM for
//         CTAs of a bandwidth-bound kernel running at the same time on another stream.
// Returns a CUDA error code (0 = launched).
int enc_gemm_launch(const CUtensorMap& ta, const CUtensorMap& tb, const EncGemmParams& p, int mode,
                    cudaStream_t stream) {
  const bool wh = mode & 1, tk = mode & 2, pair = mode & 8, compact = mode & 16;
  if (pair && (p.num_panels % 2 != 0)) return (int)cudaErrorInvalidValue;
  if (p.heads > 1 && (p.K % (p.heads * BK) != 0 || p.b_rows_per_head < p.N)) return (int)cudaErrorInvalidValue;
  if (p.units != 0) {  // ragged deal: every panel unit gets at least one range, none more ranges than there are tiles
    const int panel_units = pair ? p.num_panels / 2 : p.num_panels;
    const int base = p.units / panel_units, extra = p.units % panel_units;
    if (base < 1 || base + (extra > 0 ? 1 : 0) != p.num_splits || p.num_splits > (p.N + BN - 1) / BN)
      return (int)cudaErrorInvalidValue;
  }
  cudaError_t e;
  // 16-bit columns unless a range is too wide for them. Above k 32 the larger buffer where the epilogue is the bottleneck (an output
  // tile's MMAs take less time up to K of about 2048) or 80 entries would be cut back at nearly every step; else the longer ring.
  const int n_tiles = (p.N + BN - 1) / BN, panel_units = pair ? p.num_panels / 2 : p.num_panels;
  const int ranges = p.units != 0 ? p.units / panel_units : p.num_splits;
  const bool narrow = (n_tiles + ranges - 1) / ranges <= kNarrowTiles, large = p.K <= 2048 || p.k > 56;
  if (!tk && p.H32 != nullptr) {
    if (p.gate != nullptr || !wh) return (int)cudaErrorInvalidValue;
    e = pair ? launch_variant<true, false, 5, 0, 0, true, false, true>(ta, tb, p, stream) : launch_variant<true, false, 3, 0, 0, false, false, true>(ta, tb, p, stream);
  } else if (!tk) {
    if (pair) e = launch_variant<true, false, 6, 0, 0, true>(ta, tb, p, stream);
    else e = (mode & 4) ? launch_variant<true, false, 3, 0, 0, false>(ta, tb, p, stream)
                        : launch_variant<true, false, 4, 0, 0, false>(ta, tb, p, stream);
  } else if (p.k <= 32) {
    if (pair && !wh && narrow) e = compact ? launch_variant<false, true, 4, 32, 80, true, true>(ta, tb, p, stream)
                                           : launch_variant<false, true, 5, 32, 80, true, true>(ta, tb, p, stream);
    else if (pair) e = wh ? launch_variant<true, true, 5, 32, 64, true>(ta, tb, p, stream) : launch_variant<false, true, 5, 32, 64, true>(ta, tb, p, stream);
    else if (!wh && narrow) e = launch_variant<false, true, 3, 32, 96, false, true>(ta, tb, p, stream);
    else e = wh ? launch_variant<true, true, 3, 32, 64, false>(ta, tb, p, stream) : launch_variant<false, true, 3, 32, 64, false>(ta, tb, p, stream);
  } else {
    if (pair && !wh && narrow) e = compact ? launch_variant<false, true, 4, 64, 80, true, true>(ta, tb, p, stream)
                                   : large ? launch_variant<false, true, 4, 64, 128, true, true>(ta, tb, p, stream)
                                           : launch_variant<false, true, 5, 64, 80, true, true>(ta, tb, p, stream);
    else if (pair) e = wh ? launch_variant<true, true, 4, 64, 96, true>(ta, tb, p, stream) : launch_variant<false, true, 4, 64, 96, true>(ta, tb, p, stream);
    else if (!wh && narrow) e = launch_variant<false, true, 3, 64, 96, false, true>(ta, tb, p, stream);
    else e = wh ? launch_variant<true, true, 3, 64, 80, false>(ta, tb, p, stream) : launch_variant<false, true, 3, 64, 80, false>(ta, tb, p, stream);
  }
  return (int)e;
}

int enc_gemm_slots_for_k(int k) { return k <= 32 ? 32 : 64; }

}  // namespace lmsae
