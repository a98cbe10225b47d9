// Causal attention with separate query/key and value widths on sm_100a tensor cores (tcgen05 + TMEM + TMA).
//
// Low-rank sparse attention dictionaries (models/lorsa.py:642-661,714-725,864-904 of the reference project) run one
// attention per QK head whose value / output width is the head's OV group: q, k are [batch, seq, heads, d_qk] and
// v is [batch, seq, heads, d_v] with d_v != d_qk in general, which the flash kernels of the usual libraries do not take.
//
// Forward (attn_fwd_kernel): tiles of a 128-query block, head, value chunk of DV columns and batch element; sixteen warps, four threads
// to a query row (= TMEM lane), and one that issues the TMA loads and the MMAs.
//   per 128-key block (causal: only blocks up to the diagonal):
//     TMA      K block [128 x DQK] and V block [128 x DV] (64-column atoms, 128-byte swizzle) -> shared memory
//     tcgen05  S = Q K^T            (128 x 128 x DQK, accumulator in TMEM columns [0, 128))
//     threads  read their S row from TMEM, online softmax in the exp2 domain, write P as bf16 into shared memory in the
//              swizzled K-major layout the tensor core reads
//     tcgen05  O += P V             (128 x DV x 128, TMEM columns [128, 128 + DV))
//              (accumulating in TMEM; the rows rescale it in place only when their maximum has grown a lot)
//   epilogue: O / l as bf16, log-sum-exp per row for the backward pass.
// V is read as it is, [batch, seq, heads, d_v], as the MN-major operand of P V: no transposed copy of it exists.
// Every mbarrier wait is bounded; on expiry the CTA records a status code, stops issuing work and frees its TMEM.
#include "gather.cuh"
#include "kernels.h"

namespace lmsae {

namespace {

constexpr int ATT_BM = 128;  // queries per CTA
constexpr int ATT_BN = 128;  // keys per block
constexpr int ATOM_BYTES_128 = 128 * 128;  // 128 rows x 64 bf16

template <int DQK, int DV>
struct AttnSmem {
  static constexpr int kQOff = 0;
  static constexpr int kQBytes = (DQK / 64) * ATOM_BYTES_128;
  static constexpr int kKOff = kQOff + kQBytes;        // two K buffers
  static constexpr int kVOff = kKOff + 2 * kQBytes;    // two V buffers
  static constexpr int kVBytes = (DV / 64) * ATOM_BYTES_128;  // atoms of 128 keys x 64 columns
  static constexpr int kPOff = kVOff + 2 * kVBytes;    // two P buffers
  static constexpr int kPBytes = 2 * ATOM_BYTES_128;
  static constexpr int kXchOff = kPOff + 2 * kPBytes;  // float [2][4][128]: row statistics exchanged between column quarters
  static constexpr int kBarOff = kXchOff + 2 * 4 * 128 * 4;
  static constexpr int kNumBars = 15;
  static constexpr int kTmemPtrOff = kBarOff + kNumBars * 8;
  static constexpr int kAbortOff = kTmemPtrOff + 4;
  static constexpr int kTotal = kAbortOff + 4;
  static constexpr int kDynamicBytes = kTotal + 1024;
};

// Two-element fp32 arithmetic (one instruction for a pair): d = a * b + c and d = a + b on (lo, hi) pairs.
__device__ __forceinline__ void fma_f32x2(float& d0, float& d1, float a0, float a1, float b, float c) {
  asm("{\n\t"
      ".reg .b64 ra, rb, rc, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\t"
      "mov.b64 rb, {%4, %4};\n\t"
      "mov.b64 rc, {%5, %5};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\t"
      "mov.b64 {%0, %1}, rd;\n\t"
      "}"
      : "=f"(d0), "=f"(d1)
      : "f"(a0), "f"(a1), "f"(b), "f"(c));
}
// max of three in one instruction
__device__ __forceinline__ float max3_f32(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ void add_f32x2(float& d0, float& d1, float a0, float a1) {
  asm("{\n\t"
      ".reg .b64 ra, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\t"
      "mov.b64 rd, {%0, %1};\n\t"
      "add.rn.f32x2 rd, rd, ra;\n\t"
      "mov.b64 {%0, %1}, rd;\n\t"
      "}"
      : "+f"(d0), "+f"(d1)
      : "f"(a0), "f"(a1));
}

// byte offset of the 16-byte chunk `chunk` (0..7) of row `row` inside a 128-byte-swizzled K-major atom
__device__ __forceinline__ uint32_t sw128_chunk_off(int row, int chunk) {
  return (uint32_t)(row * 128 + ((chunk ^ (row & 7)) << 4));
}

}  // namespace

constexpr int FWD_ROW_WARPS = 16;      // warp w works on query rows 32 (w % 4) .. + 31 and key columns 32 (w / 4) .. + 31
constexpr int FWD_ROW_THREADS = FWD_ROW_WARPS * 32;
constexpr int FWD_THREADS = FWD_ROW_THREADS + 32;  // + the last warp: TMA + MMA issue
constexpr float kRescaleSlack = 8.0f;  // log2 units the running reference may lag behind the true row maximum

// Persistent: one CTA per SM walks a list of tiles (query block, head, value chunk, batch element), longest first, so
// that the loads and first MMAs of the next tile run while the softmax warps finish and store the current one.
// K, V, P (shared memory) and S (TMEM) are double-buffered over the sequence of key blocks of ALL tiles of the CTA:
// the g-th key block uses buffer g & 1 and completes phase g >> 1 of that buffer's barriers. The output accumulator is
// double-buffered over tiles (tile t uses buffer t & 1). Roles and hand-offs (mbarriers and 128-thread named barriers; no
// CTA-wide barrier inside the loops):
//   issuer   loads two key blocks ahead inside a tile; S(g+1) is computed while the rows work on S(g); P V (g) as soon
//            as P(g) is written; a K / V buffer is refilled when S / P V of its previous block has consumed it.
//   rows     four threads per query row, one per quarter of the 128 keys of a block (sixteen warps: the softmax work is
//            latency-bound, so the warps are there to hide each other's TMEM loads and barrier polls): S(g) TMEM -> 32
//            registers, release the S buffer; the four exchange their maxima through shared memory; the output accumulator stays in TMEM
//            and is only rescaled when the maximum has grown by more than 2^8 since the reference was set (rarely
//            after the first blocks), which keeps p <= 256 and the sums well inside fp32 / bf16 range; exponentials ->
//            P (bf16, swizzled K-major, two 64-key atoms) -> signal. After a tile's last block: O / l
//            to global memory, release the accumulator buffer.
template <int DQK, int DV>
__global__ void __launch_bounds__(FWD_THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const AttnParams p) {
  pdl_wait();
  using L = AttnSmem<DQK, DV>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  uint64_t* bar_q = bars + 0;
  uint64_t* bar_k = bars + 1;        // [2]
  uint64_t* bar_v = bars + 3;        // [2]
  uint64_t* bar_s_full = bars + 5;   // [2]
  uint64_t* bar_s_free = bars + 7;   // [2]
  uint64_t* bar_p_full = bars + 9;   // [2]
  uint64_t* bar_pv_done = bars + 11; // [2]
  uint64_t* bar_o_free = bars + 13;  // [2]
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem + L::kTmemPtrOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kAbortOff);

  const int warp = threadIdx.x >> 5;
  const int n_qblocks = (p.seq + ATT_BM - 1) / ATT_BM;
  const int dv_chunks = p.dv / DV;
  const int per_qblock = p.heads * dv_chunks * p.batch;  // tiles that share a query block index (same length)
  const int n_tiles = n_qblocks * per_qblock;

  if (threadIdx.x == 0) {
    mbar_init(bar_q, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&bar_k[i], 1);
      mbar_init(&bar_v[i], 1);
      mbar_init(&bar_s_full[i], 1);
      // (one arrival per softmax warp: hundreds of arrivals on one shared-memory word per key block would serialise)
      mbar_init(&bar_s_free[i], FWD_ROW_WARPS);
      mbar_init(&bar_p_full[i], FWD_ROW_WARPS);
      mbar_init(&bar_pv_done[i], 1);
      mbar_init(&bar_o_free[i], FWD_ROW_WARPS);
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == FWD_ROW_WARPS) {
    tmem_alloc(tmem_ptr_smem, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;  // S buffers at columns [0, 128) and [128, 256), O buffers at 256 and 384

  // tile w of the global list (longest query blocks first): query block, then (batch, head, value chunk)
  auto decode_tile = [&](int w, int& qblk, int& head, int& dv0, int& batch) {
    qblk = n_qblocks - 1 - w / per_qblock;
    int r = w % per_qblock;
    batch = r / (p.heads * dv_chunks);
    r -= batch * (p.heads * dv_chunks);
    head = r / dv_chunks;
    dv0 = (r - head * dv_chunks) * DV;
  };

  if (warp == FWD_ROW_WARPS) {
    // ------------------------------------------------------------------ TMA + MMA issuer
    if (elect_one()) {
      bool ok = true;
      int where = 0;
      uint32_t g0 = 0;  // key blocks issued by this CTA before the current tile
      int t = 0;
      for (int w = (int)blockIdx.x; w < n_tiles && ok; w += (int)gridDim.x, ++t) {
        int qblk, head, dv0, batch;
        decode_tile(w, qblk, head, dv0, batch);
        const int q0 = qblk * ATT_BM;
        const int n_kblocks = qblk + 1;  // causal: key blocks 0 .. diagonal
        const uint32_t tmem_o = tmem_base + 2 * ATT_BN + (uint32_t)((t & 1) * DV);
        auto load_k = [&](int kb) {
          const int u = (g0 + kb) & 1;
          mbar_arrive_expect_tx(&bar_k[u], L::kQBytes);
          for (int a = 0; a < DQK / 64; ++a)
            tma_load_3d(smem + L::kKOff + u * L::kQBytes + a * ATOM_BYTES_128, &tmap_k, &bar_k[u], head * DQK + a * 64, kb * ATT_BN, batch);
        };
        auto load_v = [&](int kb) -> bool {
          const uint32_t g = g0 + kb;
          const int u = g & 1;
          // the buffer's previous block is g - 2: its P V must have read it
          if (g >= 2 && !mbar_wait_bounded(&bar_pv_done[u], ((g - 2) >> 1) & 1, abort_flag)) return false;
          mbar_arrive_expect_tx(&bar_v[u], L::kVBytes);
          for (int a = 0; a < DV / 64; ++a)
            tma_load_3d(smem + L::kVOff + u * L::kVBytes + a * ATOM_BYTES_128, &tmap_v, &bar_v[u], head * p.dv + dv0 + a * 64, kb * ATT_BN, batch);
          return true;
        };
        auto issue_s = [&](int kb) {
          const int u = (g0 + kb) & 1;
          constexpr uint32_t idesc_s = make_idesc_bf16(ATT_BM, ATT_BN);
#pragma unroll
          for (int kk = 0; kk < DQK / 16; ++kk) {
            const uint32_t qa = smem_u32(smem + L::kQOff + (kk / 4) * ATOM_BYTES_128);
            const uint32_t ka = smem_u32(smem + L::kKOff + u * L::kQBytes + (kk / 4) * ATOM_BYTES_128);
            umma_bf16_ss(tmem_base + (uint32_t)(u * ATT_BN), make_sw128_kmajor_desc(qa) + (uint64_t)((kk % 4) * 2),
                         make_sw128_kmajor_desc(ka) + (uint64_t)((kk % 4) * 2), idesc_s, kk > 0 ? 1u : 0u);
          }
          umma_commit(&bar_s_full[u]);
        };
        // The previous tile's S MMAs have all completed (their barriers were waited for below), so Q and the K buffers
        // are free; V buffers are checked in load_v.
        where = 1;
        mbar_arrive_expect_tx(bar_q, L::kQBytes);
        for (int a = 0; a < DQK / 64; ++a)
          tma_load_3d(smem + L::kQOff + a * ATOM_BYTES_128, &tmap_q, bar_q, head * DQK + a * 64, q0, batch);
        load_k(0);
        if (n_kblocks > 1) load_k(1);
        ok = load_v(0);
        // S(0): Q and K(0) landed; the S buffer's previous block (g0 - 2) was read by the rows
        ok = ok && mbar_wait_bounded(bar_q, t & 1, abort_flag) && mbar_wait_bounded(&bar_k[g0 & 1], (g0 >> 1) & 1, abort_flag);
        if (ok && g0 >= 2) ok = mbar_wait_bounded(&bar_s_free[g0 & 1], ((g0 - 2) >> 1) & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        issue_s(0);
        // V(1) goes into the buffer that the previous tile's LAST block used: this wait is the one place where the
        // issuer depends on the rows having finished that tile's last softmax, so it comes after S(0) is under way
        where = 2;
        if (n_kblocks > 1) ok = load_v(1);
        // the accumulator buffer of this tile was last used by tile t - 2: its rows must have stored their outputs
        if (ok && t >= 2) ok = mbar_wait_bounded(&bar_o_free[t & 1], ((t - 2) >> 1) & 1, abort_flag);
        for (int kb = 0; kb < n_kblocks && ok; ++kb) {
          const uint32_t g = g0 + kb;
          const int u = g & 1;
          const uint32_t ph = (g >> 1) & 1;  // phase of this block's use of buffer u
          const bool more = kb + 1 < n_kblocks;
          if (more) {
            // S(kb+1): its K block has landed and the rows have released the S buffer it overwrites (block g - 1)
            where = 10 * kb + 3;
            ok = mbar_wait_bounded(&bar_k[u ^ 1], ((g + 1) >> 1) & 1, abort_flag);
            if (ok && g >= 1) ok = mbar_wait_bounded(&bar_s_free[u ^ 1], ((g - 1) >> 1) & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            issue_s(kb + 1);
          }
          // K buffer u is free once S(kb) has been computed: fetch block kb + 2 into it
          where = 10 * kb + 4;
          ok = mbar_wait_bounded(&bar_s_full[u], ph, abort_flag);
          if (!ok) break;
          if (kb + 2 < n_kblocks) load_k(kb + 2);
          // P V (kb)
          where = 10 * kb + 5;
          ok = mbar_wait_bounded(&bar_p_full[u], ph, abort_flag) && mbar_wait_bounded(&bar_v[u], ph, abort_flag);
          if (!ok) break;
          tc_fence_after();
          constexpr uint32_t idesc_o = make_idesc_bf16(ATT_BM, DV, false, true);
#pragma unroll
          for (int kk = 0; kk < ATT_BN / 16; ++kk) {
            const uint32_t pa = smem_u32(smem + L::kPOff + u * L::kPBytes + (kk / 4) * ATOM_BYTES_128);
            const uint32_t va = smem_u32(smem + L::kVOff + u * L::kVBytes) + kk * 2048;  // sixteen keys a step
            umma_bf16_ss(tmem_o, make_sw128_kmajor_desc(pa) + (uint64_t)((kk % 4) * 2), make_sw128_mnmajor_desc(va, ATOM_BYTES_128), idesc_o,
                         (kb > 0 || kk > 0) ? 1u : 0u);
          }
          umma_commit(&bar_pv_done[u]);
          // the V buffer of the previous block is free once its P V has completed (it ran before this one): refill it
          if (kb >= 1 && more) {
            where = 10 * kb + 6;
            ok = load_v(kb + 1);
          }
        }
        g0 += (uint32_t)n_kblocks;
      }
      if (!ok) {
        report_status(p.status, kTimeoutFullBarrier, where);
        *abort_flag = 1;
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax rows
    const int quarter = warp & 3, cq = warp >> 2, lane = (int)threadIdx.x & 31;
    const int row = quarter * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    const uint32_t s_col = (uint32_t)(cq * 32);
    // output columns of this thread (rescale and final store): a quarter of DV, at least one 32-column TMEM load
    constexpr int O_W = DV / 4 >= 32 ? DV / 4 : 32;
    const bool o_active = cq * O_W < DV;
    const uint32_t o_col = (uint32_t)(cq * O_W);
    float* xch = reinterpret_cast<float*>(smem + L::kXchOff);  // [2 parities][4 column quarters][128 rows]
    const float sc = p.scale_log2;
    bool ok = true;
    uint32_t g0 = 0;
    int t = 0;
    int w = (int)blockIdx.x;
    int met = 0;  // where a wait ran out: barriers of the row quarter that this warp came to in the tile
    for (; w < n_tiles && ok; w += (int)gridDim.x, ++t) {
      int qblk, head, dv0, batch;
      decode_tile(w, qblk, head, dv0, batch);
      const int q0 = qblk * ATT_BM;
      const int n_kblocks = qblk + 1;
      const int qpos = q0 + row;
      const bool row_ok = qpos < p.seq;
      const uint32_t tmem_o = tmem_base + 2 * ATT_BN + (uint32_t)((t & 1) * DV);
      float m_ref = -INFINITY, l_run = 0.0f;
      for (int kb = 0; kb < n_kblocks && ok; ++kb) {
        const uint32_t g = g0 + kb;
        const int u = g & 1;
        const uint32_t ph = (g >> 1) & 1;
        const int k0 = kb * ATT_BN + (int)s_col;
        // (a failed wait ends the loops for the whole warp: the TMEM accesses and votes below are warp-wide)
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bar_s_full[u], ph, abort_flag))) { ok = false; met = kb; break; }
        tc_fence_after();
        uint32_t s[32];
        tmem_ld_32x32b_x32(tmem_base + (uint32_t)(u * ATT_BN) + lane_off + s_col, s);
        tmem_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_s_free[u]);
        // masked raw scores and their maximum (only the diagonal and the last block have anything to mask)
        // (warp-uniform branch: the common, unmasked case costs one maximum per element and nothing else)
        const int last_ok = min(qpos, p.seq - 1) - k0;  // columns 0 .. last_ok of this thread's 32 are visible
        float m_raw = -INFINITY;
        if (__any_sync(0xffffffffu, last_ok < 31)) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            if (j > last_ok) s[j] = 0xff800000u;  // -inf
            m_raw = fmaxf(m_raw, __uint_as_float(s[j]));
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; j += 2) m_raw = max3_f32(m_raw, __uint_as_float(s[j]), __uint_as_float(s[j + 1]));
        }
        // the other three quarters of the row: exchange through shared memory, 128-thread barrier of the four warps
        // that share these 32 rows
        float* xr = xch + (u * 4) * ATT_BM + row;
        xr[cq * ATT_BM] = m_raw;
        asm volatile("bar.sync %0, 128;" ::"r"(1 + quarter) : "memory");
        const float m_blk = fmaxf(fmaxf(xr[0], xr[ATT_BM]), fmaxf(xr[2 * ATT_BM], xr[3 * ATT_BM])) * sc;  // sc > 0
        float alpha = 1.0f;
        bool rescale = false;
        if (m_blk > m_ref + kRescaleSlack || m_ref == -INFINITY) {
          const float m_new = fmaxf(m_ref, m_blk);
          if (m_new != -INFINITY) {
            alpha = exp2f(m_ref - m_new);  // 0 when nothing was accumulated under the old reference
            rescale = kb > 0;
            m_ref = m_new;
          }
        }
        const float m_use = (m_ref == -INFINITY) ? 0.0f : m_ref;
        if (__any_sync(0xffffffffu, rescale)) {  // this warp's share of the output columns
          // the accumulator belongs to the tensor core until P V (g - 1) has completed
          if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bar_pv_done[u ^ 1], ((g - 1) >> 1) & 1, abort_flag))) { ok = false; met = kb + 1; break; }
          tc_fence_after();
          if (o_active) {
#pragma unroll 1
            for (int c = 0; c < O_W / 32; ++c) {
              uint32_t r[32];
              tmem_ld_32x32b_x32(tmem_o + lane_off + o_col + (uint32_t)(c * 32), r);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(__uint_as_float(r[j]) * alpha);
              tmem_st_32x32b_x32(tmem_o + lane_off + o_col + (uint32_t)(c * 32), r);
            }
            tmem_wait_st();
          }
        }
        if (g >= 2) {
          // P buffer u was read by P V (g - 2)
          if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bar_pv_done[u], ((g - 2) >> 1) & 1, abort_flag))) { ok = false; met = kb + 1; break; }
        }
        l_run *= alpha;
        float l_blk = 0.0f, l_blk1 = 0.0f;
        // this quarter's 32 keys are half of a 64-key swizzle atom: 16-byte chunks (cq % 2) * 4 .. + 3 of atom cq / 2
        uint8_t* atom = smem + L::kPOff + u * L::kPBytes + (cq >> 1) * ATOM_BYTES_128;
        const float neg_m = -m_use;
#pragma unroll
        for (int gq = 0; gq < 4; ++gq) {
          float pv[8];
#pragma unroll
          for (int i = 0; i < 8; i += 2) {
            // exponent arguments and the running sums two elements per instruction; the exponentials one by one
            float a0, a1;
            fma_f32x2(a0, a1, __uint_as_float(s[gq * 8 + i]), __uint_as_float(s[gq * 8 + i + 1]), sc, neg_m);
            pv[i] = exp2f(a0);
            pv[i + 1] = exp2f(a1);
            add_f32x2(l_blk, l_blk1, pv[i], pv[i + 1]);
          }
          uint4 wv;
          wv.x = pack_bf16x2(pv[0], pv[1]);
          wv.y = pack_bf16x2(pv[2], pv[3]);
          wv.z = pack_bf16x2(pv[4], pv[5]);
          wv.w = pack_bf16x2(pv[6], pv[7]);
          *reinterpret_cast<uint4*>(atom + sw128_chunk_off(row, (cq & 1) * 4 + gq)) = wv;
        }
        l_run += l_blk + l_blk1;
        fence_proxy_async();  // the generic-proxy stores of P must be visible to the tensor core's reads
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bar_p_full[u]);
      }
      // ---- the tile's epilogue
      const uint32_t g_last = g0 + (uint32_t)n_kblocks - 1;
      if (!ok) break;
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(&bar_pv_done[g_last & 1], (g_last >> 1) & 1, abort_flag));
      if (!ok) { met = n_kblocks; break; }
      tc_fence_after();
      // total of the four partial sums; slot parity continues the per-block sequence (block g_last used g_last & 1)
      float* xl = xch + (int)((g_last + 1) & 1) * 4 * ATT_BM + row;
      xl[cq * ATT_BM] = l_run;
      asm volatile("bar.sync %0, 128;" ::"r"(1 + quarter) : "memory");
      const float l_tot = (xl[0] + xl[ATT_BM]) + (xl[2 * ATT_BM] + xl[3 * ATT_BM]);
      const float inv = l_tot > 0.0f ? 1.0f / l_tot : 0.0f;
      if (o_active) {
        __nv_bfloat16* dst = p.out + (((size_t)batch * p.seq + (row_ok ? qpos : 0)) * p.heads + head) * p.dv + dv0 + o_col;
#pragma unroll 1
        for (int c = 0; c < O_W / 32; ++c) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(tmem_o + lane_off + o_col + (uint32_t)(c * 32), r);
          tmem_wait_ld();
          if (row_ok) {
#pragma unroll
            for (int i = 0; i < 32; i += 8) {
              uint4 wv;
              wv.x = pack_bf16x2(__uint_as_float(r[i]) * inv, __uint_as_float(r[i + 1]) * inv);
              wv.y = pack_bf16x2(__uint_as_float(r[i + 2]) * inv, __uint_as_float(r[i + 3]) * inv);
              wv.z = pack_bf16x2(__uint_as_float(r[i + 4]) * inv, __uint_as_float(r[i + 5]) * inv);
              wv.w = pack_bf16x2(__uint_as_float(r[i + 6]) * inv, __uint_as_float(r[i + 7]) * inv);
              *reinterpret_cast<uint4*>(dst + c * 32 + i) = wv;
            }
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_o_free[t & 1]);
      if (row_ok && cq == 0 && p.lse != nullptr && dv0 == 0)
        p.lse[((size_t)batch * p.heads + head) * p.seq + qpos] = m_ref * 0.6931471805599453f + __logf(l_tot);
      // keep the four warps of a row quarter together across tiles: the sum exchange above and the next maximum exchange
      // use the same slots
      asm volatile("bar.sync %0, 128;" ::"r"(1 + quarter) : "memory");
      g0 += (uint32_t)n_kblocks;
    }
    if (!ok) {
      report_status(p.status, kTimeoutTmemFull, row);
      *abort_flag = 1;
      // the other warps of the quarter may have passed the wait that this one gave up at: it keeps them company at their barriers, which
      // have no limit, until they give up or are through (every warp comes to as many in a tile)
      __syncwarp();
      for (; w < n_tiles; w += (int)gridDim.x, met = 0)
        for (int left = n_qblocks - w / per_qblock + 2 - met; left > 0; --left)  // (n_kblocks and two a tile)
          asm volatile("bar.sync %0, 128;" ::"r"(1 + quarter) : "memory");
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);  // copies that may still be in flight land first
    __syncthreads();
  }
  if (warp == FWD_ROW_WARPS) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Persistent grids: one CTA per SM.
static int persistent_grid(long long tiles) {
  static const int num_sms = [] {
    int dev = 0, n = 148;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 148;
    return n;
  }();
  return (int)(tiles < num_sms ? tiles : num_sms);
}

template <int DQK, int DV>
static cudaError_t attn_fwd_variant(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                                    const AttnParams& p, cudaStream_t stream) {
  using L = AttnSmem<DQK, DV>;
  static_assert(L::kDynamicBytes <= 232448, "shared memory of one CTA exceeds 227 KB");
  auto kern = attn_fwd_kernel<DQK, DV>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynamicBytes);
  if (e != cudaSuccess) return e;
  const long long tiles = (long long)((p.seq + ATT_BM - 1) / ATT_BM) * p.heads * (p.dv / DV) * p.batch;
  if (tiles <= 0 || tiles > 2147483647LL) return cudaErrorInvalidValue;
  launch(kern, persistent_grid(tiles), FWD_THREADS, L::kDynamicBytes, stream, tq, tk, tv, p);
  return cudaGetLastError();
}

int attn_value_chunk(int dv) { return dv % 128 == 0 ? 128 : (dv % 64 == 0 ? 64 : 0); }

// =============================================================================================================
// Backward. With P = softmax(scale * Q K^T) (causal), O = P V, D = rowsum(dO * O):
//   dV = P^T dO,   dP = dO V^T,   dS = P * (dP - D),   dQ = scale * dS K,   dK = scale * dS^T Q.
// Two launches of one persistent template, attn_bwd_kernel (one CTA per SM, tiles dealt out longest first):
//   DVC 0   a tile is a query block and walks its key blocks:   dQ += dS K
//   else    a tile is a key block (and value chunk) and walks its query blocks:   dV += P^T dO,  dK += dS^T Q
// In both, every step computes S = Q K^T and dP = dO V^T of one 128 x 128 block with queries in the TMEM lanes, so that the row
// statistics are one value per thread, and every operand is read from the row-major tensors: where a product contracts over
// positions its tile is a MN-major operand of the same shared-memory copy (P and dS as MN-major A, Q, K and dO as MN-major B), so
// that no transposed copies of Q, K, dO and V exist.
//   warps 0-15  softmax rows: four threads per query row, 32 key columns each. S and dP go from TMEM to registers at once, which
//               frees both buffers: the tensor core computes the next block's while these warps work on exponentials. P and
//               dS (bf16, two 64-key swizzle atoms) are kept packed in registers until the MMAs of the previous block have read the buffer.
//   warp 16     TMA producer; warp 17 the MMA issuer: S(g), dP(g), then the accumulating products of block g - 1
// A finished tile is stored one block late (after the first block of the next tile), so that nothing waits for its last product.
// What bounds a block: 1024 cycles of exponentials (16 a cycle and SM) against 1024 (dQ) or 1536 (dK/dV) cycles of MMAs at
// d_qk 64, d_v 128; measured about 3400 and 5300 (4608 blocks on 148 CTAs at the size below): hand-offs between the three roles. The tensor
// pipe is active 34 and 30 % of the time, the exponential pipe 36 and 22 %.
// 2 x 64 heads x 1024 positions, d_qk 64, d_v 128: dQ 146 -> 61 us, dK/dV 226 -> 97 us against kernels of four warps that took turns with
// the tensor core, and about 250 us of transposed copies and conversions around them are gone.
// =============================================================================================================
namespace {

// D[tmem] (+)= A * B^T over 16 * steps of K, both tiles K-major, made of 64-column swizzle atoms `a_atom` / `b_atom` bytes apart.
__device__ __forceinline__ void issue_mma_atoms(uint32_t tmem_d, uint32_t a_base, uint32_t a_atom, uint32_t b_base,
                                                uint32_t b_atom, int steps, uint32_t idesc, bool accumulate) {
  for (int kk = 0; kk < steps; ++kk) {
    const uint64_t da = make_sw128_kmajor_desc(a_base + (uint32_t)(kk / 4) * a_atom) + (uint64_t)((kk % 4) * 2);
    const uint64_t db = make_sw128_kmajor_desc(b_base + (uint32_t)(kk / 4) * b_atom) + (uint64_t)((kk % 4) * 2);
    umma_bf16_ss(tmem_d, da, db, idesc, (accumulate || kk > 0) ? 1u : 0u);
  }
}

constexpr int BWD_THREADS = FWD_ROW_THREADS + 64;  // sixteen row warps, the producer and the issuer
constexpr int AB = ATOM_BYTES_128;

// Shared memory of both kernels in atoms of 128 rows x 64 columns. FIX: the pair of tiles a CTA keeps for a whole tile (Q and dO, or
// K and V), WALK: the ones that change from block to block. A walking Q / K tile is in use from its S to the accumulating product of
// its block, one block later: three buffers keep the loads ahead. Fixed value tiles wider than two atoms are streamed through
// their two slots, once per block.
template <int DQK, bool DKV>
struct BwdSmem {
  static constexpr int kQkAtoms = DQK / 64;
  static constexpr int kFixBufs = DQK == 64 && !DKV ? 2 : 1;
  static constexpr int kWalkBufs = DQK == 64 ? 3 : (DKV ? 1 : 2);
  static constexpr int kFixValSlots = 2, kWalkValSlots = 4;
  static constexpr int kFixOff = 0;
  static constexpr int kWalkOff = kFixOff + kFixBufs * kQkAtoms * AB;
  static constexpr int kFixValOff = kWalkOff + kWalkBufs * kQkAtoms * AB;
  static constexpr int kWalkValOff = kFixValOff + kFixValSlots * AB;
  static constexpr int kDsOff = kWalkValOff + kWalkValSlots * AB;
  static constexpr int kPOff = kDsOff + 2 * AB;
  static constexpr int kBarOff = kPOff + (DKV ? 2 * AB : 0);
  static constexpr int kNumBars = 2 * (kFixBufs + kWalkBufs + kFixValSlots + kWalkValSlots) + 6;
  static constexpr int kTmemPtrOff = kBarOff + kNumBars * 8;
  static constexpr int kAbortOff = kTmemPtrOff + 4;
  static constexpr int kDynamicBytes = kAbortOff + 4 + 1024;
};

struct BwdBars {
  uint64_t *fix_full, *fix_free, *walk_full, *walk_free, *fval_full, *fval_free, *wval_full, *wval_free;
  uint64_t *sdp_full;  // S and dP of a block are in TMEM
  uint64_t *sdp_free;  // the rows have read them
  uint64_t *out_full;  // the rows have written dS (and P)
  uint64_t *out_free;  // the block's accumulating products are done
  uint64_t *acc_free;  // [2] the rows have stored a finished tile
};

template <class L>
__device__ __forceinline__ BwdBars bwd_bars(uint8_t* smem) {
  uint64_t* b = reinterpret_cast<uint64_t*>(smem + L::kBarOff);
  BwdBars r;
  r.fix_full = b; b += L::kFixBufs;
  r.fix_free = b; b += L::kFixBufs;
  r.walk_full = b; b += L::kWalkBufs;
  r.walk_free = b; b += L::kWalkBufs;
  r.fval_full = b; b += L::kFixValSlots;
  r.fval_free = b; b += L::kFixValSlots;
  r.wval_full = b; b += L::kWalkValSlots;
  r.wval_free = b; b += L::kWalkValSlots;
  r.sdp_full = b; r.sdp_free = b + 1; r.out_full = b + 2; r.out_free = b + 3; r.acc_free = b + 4;
  return r;
}

// One block's share of a thread: 32 key columns of its query row -> P and dS (unscaled), packed to bf16 pairs.
// `last`: columns 0 .. last are visible (31 or more: all of them).
template <bool WANT_P, bool MASK>
__device__ __forceinline__ void bwd_columns(const uint32_t (&rs)[32], const uint32_t (&rp)[32], float scale_log2, float neg_lse2, float neg_delta,
                                            int last, uint32_t (&pk)[16], uint32_t (&dk)[16]) {
#pragma unroll
  for (int j = 0; j < 32; j += 2) {
    float a0, a1, d0 = neg_delta, d1 = neg_delta;
    fma_f32x2(a0, a1, __uint_as_float(rs[j]), __uint_as_float(rs[j + 1]), scale_log2, neg_lse2);
    float p0 = exp2f(a0), p1 = exp2f(a1);
    add_f32x2(d0, d1, __uint_as_float(rp[j]), __uint_as_float(rp[j + 1]));
    if constexpr (MASK) {
      if (j > last) { p0 = 0.0f; d0 = 0.0f; }
      if (j + 1 > last) { p1 = 0.0f; d1 = 0.0f; }
    }
    if constexpr (WANT_P) pk[j / 2] = pack_bf16x2(p0, p1);
    dk[j / 2] = pack_bf16x2(p0 * d0, p1 * d1);
  }
}
template <bool WANT_P>
__device__ __forceinline__ void bwd_block(const uint32_t (&rs)[32], const uint32_t (&rp)[32], float scale_log2, float neg_lse2, float neg_delta,
                                          int last, uint32_t (&pk)[16], uint32_t (&dk)[16]) {
  // (only the diagonal and the last block have anything to mask: the branch is the same for the whole warp)
  if (__any_sync(0xffffffffu, last < 31)) bwd_columns<WANT_P, true>(rs, rp, scale_log2, neg_lse2, neg_delta, last, pk, dk);
  else bwd_columns<WANT_P, false>(rs, rp, scale_log2, neg_lse2, neg_delta, last, pk, dk);
}

// 32 packed columns of a row to its two-atom tile: 16-byte chunks (cq % 2) * 4 .. + 3 of atom cq / 2.
__device__ __forceinline__ void bwd_store(uint8_t* tile, int row, int cq, const uint32_t (&v)[16]) {
  uint8_t* atom = tile + (cq >> 1) * AB;
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<uint4*>(atom + sw128_chunk_off(row, (cq & 1) * 4 + i)) = make_uint4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
}

// 32 accumulator columns of a thread's lane, times `mul`, to global memory (fp32, or bf16 in one rounding).
__device__ __forceinline__ void bwd_emit(uint32_t taddr, float mul, void* base, size_t offset, bool bf16_out, bool row_ok) {
  uint32_t r[32];
  tmem_ld_32x32b_x32(taddr, r);
  tmem_wait_ld();
  if (!row_ok) return;
  if (bf16_out) {
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(base) + offset;
#pragma unroll
    for (int i = 0; i < 32; i += 8)
      *reinterpret_cast<uint4*>(dst + i) =
          make_uint4(pack_bf16x2(__uint_as_float(r[i]) * mul, __uint_as_float(r[i + 1]) * mul),
                     pack_bf16x2(__uint_as_float(r[i + 2]) * mul, __uint_as_float(r[i + 3]) * mul),
                     pack_bf16x2(__uint_as_float(r[i + 4]) * mul, __uint_as_float(r[i + 5]) * mul),
                     pack_bf16x2(__uint_as_float(r[i + 6]) * mul, __uint_as_float(r[i + 7]) * mul));
  } else {
    float* dst = reinterpret_cast<float*>(base) + offset;
#pragma unroll
    for (int i = 0; i < 32; i += 4)
      *reinterpret_cast<float4*>(dst + i) = make_float4(__uint_as_float(r[i]) * mul, __uint_as_float(r[i + 1]) * mul,
                                                        __uint_as_float(r[i + 2]) * mul, __uint_as_float(r[i + 3]) * mul);
  }
}

}  // namespace

// DVC: value columns of a tile's dV (dK/dV kernel; its chunks other than the first leave dK alone), 0 for the dQ kernel.
template <int DQK, int DVC>
__global__ void __launch_bounds__(BWD_THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do, const AttnBwdParams p) {
  pdl_wait();
  constexpr bool DKV = DVC != 0;
  using L = BwdSmem<DQK, DKV>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const BwdBars B = bwd_bars<L>(smem);
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem + L::kTmemPtrOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::kAbortOff);
  constexpr int QK_BYTES = L::kQkAtoms * AB;

  const int warp = threadIdx.x >> 5;
  const int n_blocks = (p.seq + 127) / 128;
  const int chunks = DKV ? p.dv / (DKV ? DVC : 1) : 1;
  const int per_block = p.heads * chunks * p.batch;
  const int n_tiles = n_blocks * per_block;
  const int dv_atoms = p.dv / 64;
  const bool stream_fix = dv_atoms > L::kFixValSlots;  // the fixed value tile does not fit: once per block instead

  if (threadIdx.x == 0) {
    for (uint64_t* b = B.fix_full; b < B.fix_full + L::kNumBars; ++b)
      mbar_init(b, b == B.sdp_free || b == B.out_full || b >= B.acc_free ? FWD_ROW_WARPS : 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == FWD_ROW_WARPS + 1) {
    tmem_alloc(tmem_ptr_smem, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  const uint32_t tmem_s = tmem_base, tmem_dp = tmem_base + 128, tmem_acc = tmem_base + 256;  // acc: dQ of two tiles, or dV and dK

  // tile w: the block it belongs to (those with the longest walks first), then batch, head, value chunk
  struct Tile { int blk, head, chunk, batch, first, steps; };
  auto decode = [&](int w) {
    Tile t;
    const int i = w / per_block;
    int r = w - i * per_block;
    t.batch = r / (p.heads * chunks);
    r -= t.batch * (p.heads * chunks);
    t.head = r / chunks;
    t.chunk = r - t.head * chunks;
    t.blk = DKV ? i : n_blocks - 1 - i;
    t.first = DKV ? t.blk : 0;                          // first block of the walk
    t.steps = DKV ? n_blocks - t.blk : t.blk + 1;
    return t;
  };
  // order in which a block's value atoms are used: the chunk's own last (they stay for dV)
  auto atom_at = [&](const Tile& t, int i) {
    if constexpr (!DKV) return i;
    const int a = t.chunk * (DVC / 64) + DVC / 64 + i;
    return a < dv_atoms ? a : a - dv_atoms;
  };

  if (warp == FWD_ROW_WARPS) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      const CUtensorMap* m_fix = DKV ? &tmap_k : &tmap_q;
      const CUtensorMap* m_walk = DKV ? &tmap_q : &tmap_k;
      const CUtensorMap* m_fval = DKV ? &tmap_v : &tmap_do;
      const CUtensorMap* m_wval = DKV ? &tmap_do : &tmap_v;
      uint32_t t = 0, g = 0, nf = 0, nw = 0;
      bool ok = true;
      for (int w = (int)blockIdx.x; w < n_tiles && ok; w += (int)gridDim.x, ++t) {
        const Tile T = decode(w);
        auto load_qk = [&](const CUtensorMap* m, uint8_t* dst, uint64_t* bar, int blk) {
          mbar_arrive_expect_tx(bar, QK_BYTES);
          for (int a = 0; a < L::kQkAtoms; ++a) tma_load_3d(dst + a * AB, m, bar, T.head * DQK + a * 64, blk * 128, T.batch);
        };
        auto load_val = [&](const CUtensorMap* m, uint8_t* dst, uint64_t* bar, int atom, int blk) {
          mbar_arrive_expect_tx(bar, AB);
          tma_load_3d(dst, m, bar, T.head * p.dv + atom * 64, blk * 128, T.batch);
        };
        const uint32_t fb = t % L::kFixBufs;
        ok = mbar_wait_bounded(&B.fix_free[fb], ((t / L::kFixBufs) & 1) ^ 1, abort_flag);
        if (!ok) break;
        load_qk(m_fix, smem + L::kFixOff + fb * QK_BYTES, &B.fix_full[fb], T.blk);
        for (int s = 0; s < T.steps && ok; ++s, ++g) {
          const uint32_t wb = g % L::kWalkBufs;
          ok = mbar_wait_bounded(&B.walk_free[wb], ((g / L::kWalkBufs) & 1) ^ 1, abort_flag);
          if (!ok) break;
          load_qk(m_walk, smem + L::kWalkOff + wb * QK_BYTES, &B.walk_full[wb], T.first + s);
          for (int i = 0; i < dv_atoms && ok; ++i) {
            const int a = atom_at(T, i);
            if (stream_fix || s == 0) {
              const uint32_t slot = stream_fix ? nf & 1 : (uint32_t)i, use = stream_fix ? nf >> 1 : t;
              ok = mbar_wait_bounded(&B.fval_free[slot], (use & 1) ^ 1, abort_flag);
              if (!ok) break;
              load_val(m_fval, smem + L::kFixValOff + slot * AB, &B.fval_full[slot], a, T.blk);
              ++nf;
            }
            const uint32_t slot = nw % L::kWalkValSlots;
            ok = mbar_wait_bounded(&B.wval_free[slot], ((nw / L::kWalkValSlots) & 1) ^ 1, abort_flag);
            if (!ok) break;
            load_val(m_wval, smem + L::kWalkValOff + slot * AB, &B.wval_full[slot], a, T.first + s);
            ++nw;
          }
        }
      }
      if (!ok) {
        report_status(p.status, kTimeoutEmptyBarrier, (int)g);
        *abort_flag = 1;
      }
    }
  } else if (warp == FWD_ROW_WARPS + 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_bf16(128, 128);
      uint32_t t = 0, g = 0, nf = 0, nw = 0;
      bool ok = true;
      // the block whose accumulating products are still to be issued
      bool pending = false;
      uint32_t pg = 0, pt = 0, pval = 0;  // its index, its tile's, the slot of the first atom of its value chunk
      int ps = 0;
      bool pdk = false;
      // Block g's accumulating products follow the S and dP of block g + 1, so that the tensor core has work while the rows are at block
      // g; they come before them where the tiles that block g holds on to leave no room for those of block g + 1.
      const bool early = L::kWalkBufs == 1 || (DKV && dv_atoms + DVC / 64 > L::kWalkValSlots);
      auto accumulate = [&]() -> bool {
        if (!pending) return true;
        pending = false;
        if (ps == 0) {  // the accumulator's previous tile has been stored
          const uint32_t buf = DKV ? 0 : pt & 1, use = DKV ? pt : pt >> 1;
          if (!mbar_wait_bounded(&B.acc_free[buf], (use & 1) ^ 1, abort_flag)) return false;
        }
        if (!mbar_wait_bounded(B.out_full, pg & 1, abort_flag)) return false;
        tc_fence_after();
        const uint32_t walk = smem_u32(smem + L::kWalkOff + (pg % L::kWalkBufs) * QK_BYTES);
        const uint32_t ds = smem_u32(smem + L::kDsOff);
        if constexpr (!DKV) {
          const uint32_t d = tmem_acc + (pt & 1) * DQK;
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)  // sixteen keys a step
            umma_bf16_ss(d, make_sw128_kmajor_desc(ds + (kk / 4) * AB) + (uint64_t)((kk % 4) * 2), make_sw128_mnmajor_desc(walk + kk * 2048, AB),
                         make_idesc_bf16(128, DQK, false, true), (ps > 0 || kk > 0) ? 1u : 0u);
        } else {
          const uint32_t pm = smem_u32(smem + L::kPOff), val = smem_u32(smem + L::kWalkValOff + pval * AB);
#pragma unroll
          for (int kk = 0; kk < 8; ++kk)  // sixteen queries a step
            umma_bf16_ss(tmem_acc, make_sw128_mnmajor_desc(pm + kk * 2048, AB), make_sw128_mnmajor_desc(val + kk * 2048, AB),
                         make_idesc_bf16(128, DVC, true, true), (ps > 0 || kk > 0) ? 1u : 0u);
          for (int i = 0; i < DVC / 64; ++i) umma_commit(&B.wval_free[pval + i]);
          if (pdk) {
#pragma unroll
            for (int kk = 0; kk < 8; ++kk)
              umma_bf16_ss(tmem_acc + 128, make_sw128_mnmajor_desc(ds + kk * 2048, AB), make_sw128_mnmajor_desc(walk + kk * 2048, AB),
                           make_idesc_bf16(128, DQK, true, true), (ps > 0 || kk > 0) ? 1u : 0u);
          }
        }
        umma_commit(&B.walk_free[pg % L::kWalkBufs]);
        umma_commit(B.out_free);
        return true;
      };
      for (int w = (int)blockIdx.x; w < n_tiles && ok; w += (int)gridDim.x, ++t) {
        const Tile T = decode(w);
        const uint32_t fb = t % L::kFixBufs;
        for (int s = 0; s < T.steps; ++s, ++g) {
          if (early && !(ok = accumulate())) break;
          const uint32_t wb = g % L::kWalkBufs;
          ok = (s > 0 || mbar_wait_bounded(&B.fix_full[fb], (t / L::kFixBufs) & 1, abort_flag)) &&
               mbar_wait_bounded(&B.walk_full[wb], (g / L::kWalkBufs) & 1, abort_flag) &&
               mbar_wait_bounded(B.sdp_free, (g & 1) ^ 1, abort_flag);  // the rows have read block g - 1
          if (!ok) break;
          tc_fence_after();
          const uint32_t fix = smem_u32(smem + L::kFixOff + fb * QK_BYTES), walk = smem_u32(smem + L::kWalkOff + wb * QK_BYTES);
          issue_mma_atoms(tmem_s, DKV ? walk : fix, AB, DKV ? fix : walk, AB, DQK / 16, idesc_s, false);
          const bool last = s + 1 == T.steps;
          if (last) umma_commit(&B.fix_free[fb]);
          uint32_t first_kept = 0;
          for (int i = 0; i < dv_atoms; ++i) {
            const uint32_t fslot = stream_fix ? nf & 1 : (uint32_t)i, fuse = stream_fix ? nf >> 1 : t;
            const uint32_t wslot = nw % L::kWalkValSlots;
            if (stream_fix || s == 0) ok = mbar_wait_bounded(&B.fval_full[fslot], fuse & 1, abort_flag);
            ok = ok && mbar_wait_bounded(&B.wval_full[wslot], (nw / L::kWalkValSlots) & 1, abort_flag);
            if (!ok) break;
            tc_fence_after();
            const uint32_t fv = smem_u32(smem + L::kFixValOff + fslot * AB), wv = smem_u32(smem + L::kWalkValOff + wslot * AB);
            issue_mma_atoms(tmem_dp, DKV ? wv : fv, 0, DKV ? fv : wv, 0, 4, idesc_s, i > 0);
            if (stream_fix || last) umma_commit(&B.fval_free[fslot]);
            const bool kept = DKV && i >= dv_atoms - DVC / 64;  // (needed once more, for dV)
            if (!kept) umma_commit(&B.wval_free[wslot]);
            if (DKV && i == dv_atoms - DVC / 64) first_kept = wslot;
            if (stream_fix) ++nf;
            ++nw;
          }
          if (!ok) break;
          umma_commit(B.sdp_full);
          if (!early && !(ok = accumulate())) break;
          pending = true;
          pg = g; pt = t; ps = s; pval = first_kept; pdk = T.chunk == 0;
        }
      }
      ok = ok && accumulate();
      if (!ok) {
        report_status(p.status, kTimeoutFullBarrier, (int)g);
        *abort_flag = 1;
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax rows
    const int quarter = warp & 3, cq = warp >> 2, lane = (int)threadIdx.x & 31;
    const int row = quarter * 32 + lane;
    const uint32_t lane_off = (uint32_t)(quarter * 32) << 16;
    bool ok = true;
    uint32_t g = 0, t = 0;
    // a finished tile that is still to be stored
    bool pending = false;
    Tile pT{};
    uint32_t pt = 0;
    auto store_tile = [&]() {  // (its last accumulating product has completed)
      tc_fence_after();
      const int pos = pT.blk * 128 + row;
      const bool row_ok = pos < p.seq;
      const size_t at = ((size_t)pT.batch * p.seq + (row_ok ? pos : 0)) * p.heads + pT.head;
      if constexpr (!DKV) {
        if (cq < DQK / 32)
          bwd_emit(tmem_acc + (pt & 1) * DQK + lane_off + cq * 32, p.scale, p.dq, at * DQK + cq * 32, p.bf16_out, row_ok);
      } else {
        if (cq < DVC / 32)
          bwd_emit(tmem_acc + lane_off + cq * 32, 1.0f, p.dv_out, at * p.dv + pT.chunk * DVC + cq * 32, p.bf16_out, row_ok);
        if (pT.chunk == 0 && cq < DQK / 32)
          bwd_emit(tmem_acc + 128 + lane_off + cq * 32, p.scale, p.dk, at * DQK + cq * 32, p.bf16_out, row_ok);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&B.acc_free[DKV ? 0 : pt & 1]);
      pending = false;
    };
    for (int w = (int)blockIdx.x; w < n_tiles && ok; w += (int)gridDim.x, ++t) {
      const Tile T = decode(w);
      const size_t stat0 = ((size_t)T.batch * p.heads + T.head) * p.seq;
      auto load_stats = [&](int qblk, float& nl, float& nd) {
        const int qpos = qblk * 128 + row;
        const bool in = qpos < p.seq;
        nl = in ? -p.lse[stat0 + qpos] * 1.4426950408889634f : -INFINITY;  // (no position: every probability of the row is 0)
        nd = in ? -p.delta[stat0 + qpos] : 0.0f;
      };
      float neg_lse2, neg_delta;
      load_stats(DKV ? T.first : T.blk, neg_lse2, neg_delta);
      for (int s = 0; s < T.steps; ++s, ++g) {
        const int qblk = DKV ? T.first + s : T.blk, kblk = DKV ? T.blk : T.first + s;
        float next_lse2 = neg_lse2, next_delta = neg_delta;
        if (DKV && s + 1 < T.steps) load_stats(qblk + 1, next_lse2, next_delta);
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(B.sdp_full, g & 1, abort_flag));
        if (!ok) break;
        tc_fence_after();
        uint32_t pk[16], dk[16];
        {
          uint32_t rs[32], rp[32];
          tmem_ld_32x32b_x32(tmem_s + lane_off + (uint32_t)(cq * 32), rs);
          tmem_ld_32x32b_x32(tmem_dp + lane_off + (uint32_t)(cq * 32), rp);
          tmem_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(B.sdp_free);
          const int last = min(qblk * 128 + row, p.seq - 1) - (kblk * 128 + cq * 32);
          bwd_block<DKV>(rs, rp, p.scale_log2, neg_lse2, neg_delta, last, pk, dk);
        }
        // the previous block's accumulating products have read P and dS
        ok = __all_sync(0xffffffffu, mbar_wait_bounded(B.out_free, (g & 1) ^ 1, abort_flag));
        if (!ok) break;
        bwd_store(smem + L::kDsOff, row, cq, dk);
        if constexpr (DKV) bwd_store(smem + L::kPOff, row, cq, pk);
        fence_proxy_async();  // the generic-proxy stores must be visible to the tensor core's reads
        __syncwarp();
        if (lane == 0) mbar_arrive(B.out_full);
        if (pending) store_tile();  // (s == 0: the tile before this one, whose last products have just been waited for)
        neg_lse2 = next_lse2;
        neg_delta = next_delta;
      }
      if (!ok) break;
      pending = true;
      pT = T;
      pt = t;
    }
    if (ok && pending) {
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(B.out_free, (g & 1) ^ 1, abort_flag));
      if (ok) store_tile();
    }
    if (!ok) {
      report_status(p.status, kTimeoutTmemFull, row);
      *abort_flag = 1;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);  // copies that may still be in flight land first
    __syncthreads();
  }
  if (warp == FWD_ROW_WARPS + 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

template <int DQK, int DVC>
static cudaError_t attn_bwd_variant(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo,
                                    const AttnBwdParams& p, cudaStream_t stream) {
  using L = BwdSmem<DQK, DVC != 0>;
  static_assert(L::kDynamicBytes <= 232448, "shared memory of one CTA exceeds 227 KB");
  auto kern = attn_bwd_kernel<DQK, DVC>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kDynamicBytes);
  if (e != cudaSuccess) return e;
  const long long tiles = (long long)((p.seq + 127) / 128) * p.heads * (DVC != 0 ? p.dv / (DVC != 0 ? DVC : 1) : 1) * p.batch;
  if (tiles <= 0 || tiles > 2147483647LL) return cudaErrorInvalidValue;
  launch(kern, persistent_grid(tiles), BWD_THREADS, L::kDynamicBytes, stream, tq, tk, tv, tdo, p);
  return cudaGetLastError();
}

int attn_bwd_launch(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tdo, const AttnBwdParams& p,
                    cudaStream_t stream) {
  const int dvc = attn_value_chunk(p.dv);
  if (dvc == 0 || (p.dqk != 64 && p.dqk != 128) || p.seq % 8 != 0 || p.batch > 65535 || p.heads * (p.dv / dvc) > 65535)
    return (int)cudaErrorInvalidValue;
  cudaError_t e = p.dqk == 64 ? attn_bwd_variant<64, 0>(tq, tk, tv, tdo, p, stream) : attn_bwd_variant<128, 0>(tq, tk, tv, tdo, p, stream);
  if (e != cudaSuccess) return (int)e;
  if (p.dqk == 64) e = dvc == 128 ? attn_bwd_variant<64, 128>(tq, tk, tv, tdo, p, stream) : attn_bwd_variant<64, 64>(tq, tk, tv, tdo, p, stream);
  else e = dvc == 128 ? attn_bwd_variant<128, 128>(tq, tk, tv, tdo, p, stream) : attn_bwd_variant<128, 64>(tq, tk, tv, tdo, p, stream);
  return (int)e;
}

// delta[b, h, s] = sum over the value columns of dO * O: eight lanes per (position, head), two 16-byte loads a lane and tensor at once.
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ out, long long rows, int seq, int heads, int dv,
                  float* __restrict__ delta) {
  pdl_wait();
  const int sub = threadIdx.x & 7;
  const long long r = (long long)blockIdx.x * 32 + (threadIdx.x >> 3);
  float s = 0.0f;
  if (r < rows) {
    for (int c = sub * 8; c < dv; c += 128) {  // (dv is a multiple of 8)
      const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
      const bool two = c + 64 < dv;
      const uint4 a0 = __ldg(reinterpret_cast<const uint4*>(dout + r * dv + c)), b0 = __ldg(reinterpret_cast<const uint4*>(out + r * dv + c));
      const uint4 a1 = two ? __ldg(reinterpret_cast<const uint4*>(dout + r * dv + c + 64)) : zero;
      const uint4 b1 = two ? __ldg(reinterpret_cast<const uint4*>(out + r * dv + c + 64)) : zero;
      float x[8], y[8];
      bf16x8_to_float(a0, x);
      bf16x8_to_float(b0, y);
#pragma unroll
      for (int i = 0; i < 8; ++i) s = fmaf(x[i], y[i], s);
      bf16x8_to_float(a1, x);
      bf16x8_to_float(b1, y);
#pragma unroll
      for (int i = 0; i < 8; ++i) s = fmaf(x[i], y[i], s);
    }
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (r < rows && sub == 0) {
    const long long pos = r / heads;
    delta[((pos / seq) * heads + r % heads) * seq + pos % seq] = s;
  }
}

int attn_delta_launch(const __nv_bfloat16* dout, const __nv_bfloat16* out, int batch, int seq, int heads, int dv, float* delta, cudaStream_t stream) {
  const long long rows = (long long)batch * seq * heads;
  if (rows == 0) return 0;
  launch(attn_delta_kernel, (int)((rows + 31) / 32), 256, 0, stream, dout, out, rows, seq, heads, dv, delta);
  return (int)cudaGetLastError();
}

// Value columns per CTA of the forward kernel: with 128-wide queries the double-buffered tiles only fit for 64.
int attn_fwd_value_chunk(int dqk, int dv) {
  const int c = attn_value_chunk(dv);
  return (dqk == 128 && c == 128) ? 64 : c;
}

int attn_fwd_launch(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const AttnParams& p,
                    cudaStream_t stream) {
  const int dvc = attn_fwd_value_chunk(p.dqk, p.dv);
  if (dvc == 0 || (p.dqk != 64 && p.dqk != 128) || p.seq % 8 != 0 || p.batch > 65535 || p.heads * (p.dv / dvc) > 65535)
    return (int)cudaErrorInvalidValue;
  cudaError_t e;
  if (p.dqk == 64) e = dvc == 128 ? attn_fwd_variant<64, 128>(tq, tk, tv, p, stream) : attn_fwd_variant<64, 64>(tq, tk, tv, p, stream);
  else e = attn_fwd_variant<128, 64>(tq, tk, tv, p, stream);
  return (int)e;
}

}  // namespace lmsae
