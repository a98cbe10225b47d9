// Threshold gradient of a JumpReLU head as the epilogue of its product (sm_100a):
//
//     dtheta[f] += -theta_f / window * sum over tokens b inside the window of ( G[b, f] / n_f + add_per_hit ),
//     G = d x_hat . W_D^T,   inside: x = S[b, f] * n_f > 0 and |x - theta_f| < window / 2
//
// (the straight-through gradient of activation_functions.py:15-64 in the reference project; S the summed pre-activations in bf16, n_f the
// norm of the head's decoder row). The window covers most positive pre-activations, so that G is needed densely, but only inside this
// sum: G is never written.
//
// The product is taken with FEATURES as its rows: a TMEM lane is a feature, an epilogue thread keeps its feature's norm and threshold
// in registers and walks the tokens (columns) with its sum in a register; there is no reduction over lanes, and one atomic addition
// per thread and tile ends it. S arrives by TMA beside the operands, [token][feature] as it lies in memory: lanes read
// neighbouring features of one token.
//   CTA pair (cta_group::2): 256 features x 256 tokens a tile, operands as in encoder_gemm.cu (each CTA its 128 features and half of
//   the token rows); persistent, the (panel, token tile) list is dealt round, panel-major: at any time the pairs are at a few neighbouring
//   panels, whose W_D rows come from memory once, and the d x_hat rows stay in L2 (with a contiguous share per pair all pairs' own panels
//   have to stay there too: d 2304 took 300 us instead of 209).
//   warp 0 TMA (operands and S), warp 1 MMA issuer, warp 2 TMEM, warps 4-11 epilogue: two warps per 32 features, half of the tokens each
// What bounds it: the MMAs (d 768: 6144 cycles a tile against some 2500 of the epilogue). One head of 98304 features, d 768, 4096 tokens,
// which as a product with stored G and a pass over G and S took 480 + 305 us: 446 us; 18432 features, d 2304: 225 + 97 -> 209; 30000
// features, d 256, 2000 tokens: 61 + 93 -> 72.
#include "common.cuh"
#include "kernels.h"

namespace lmsae {

namespace {

constexpr int WG_BK = 64;
constexpr int WG_STAGES = 5;
constexpr int WG_OPERAND = 128 * WG_BK * 2;      // 16 KB: 128 rows of one operand
constexpr int WG_STAGE = 2 * WG_OPERAND;
constexpr int WG_S_CHUNK = 128 * 64 * 2;         // 128 tokens x 64 features of S
constexpr int WG_TOKENS = 256;                   // tokens of a tile
constexpr int WG_EPI_WARPS = 8;
constexpr int WG_THREADS = 128 + 32 * WG_EPI_WARPS;
constexpr int WG_S_OFF = WG_STAGES * WG_STAGE;
constexpr int WG_BAR_OFF = WG_S_OFF + 4 * WG_S_CHUNK;
constexpr int WG_NUM_BARS = 2 * WG_STAGES + 4 + 8;
constexpr int WG_TMEM_PTR_OFF = WG_BAR_OFF + WG_NUM_BARS * 8;
constexpr int WG_ABORT_OFF = WG_TMEM_PTR_OFF + 4;
constexpr int WG_SMEM = WG_ABORT_OFF + 4 + 1024;
static_assert(WG_SMEM <= 232448, "shared memory of one CTA exceeds 227 KB");

}  // namespace

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(WG_THREADS, 1)
window_grad_gemm_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_g,
                        const __grid_constant__ CUtensorMap tmap_s, const WindowGradParams p) {
  pdl_wait();
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + WG_BAR_OFF);
  uint64_t* empty_bar = full_bar + WG_STAGES;
  uint64_t* acc_full = empty_bar + WG_STAGES;  // [2]
  uint64_t* acc_empty = acc_full + 2;          // [2]
  uint64_t* s_full = acc_empty + 2;            // [4] chunk (token half * 2 + feature half)
  uint64_t* s_empty = s_full + 4;              // [4]
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem + WG_TMEM_PTR_OFF);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + WG_ABORT_OFF);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();
  const bool leader = cta_rank == 0;
  const int pair = (int)(blockIdx.x >> 1), n_pairs = (int)(gridDim.x >> 1);
  const int token_tiles = (p.B + WG_TOKENS - 1) / WG_TOKENS;
  const long long n_tiles = (long long)((p.F + 255) / 256) * token_tiles;
  const int num_k = (p.d + WG_BK - 1) / WG_BK;

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * WG_STAGES + 2; ++i) mbar_init(&full_bar[i], 1);                       // stages, accumulators full
    for (int i = 0; i < 2; ++i) mbar_init(&acc_empty[i], 2 * WG_EPI_WARPS);                       // epilogue warps of both CTAs
    for (int i = 0; i < 4; ++i) mbar_init(&s_full[i], 1);
    for (int i = 0; i < 4; ++i) mbar_init(&s_empty[i], 2);                                        // the two warps that read a chunk
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&tmap_w);
    prefetch_tensormap(&tmap_g);
    prefetch_tensormap(&tmap_s);
  }
  if (warp == 2) {
    tmem_alloc_pair(tmem_ptr_smem, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer
    if (elect_one()) {
      uint32_t it = 0, lt = 0;
      bool ok = true;
      for (long long t = pair; t < n_tiles && ok; t += n_pairs, ++lt) {
        const int f0 = (int)(t / token_tiles) * 256 + (int)cta_rank * 128, b0 = (int)(t % token_tiles) * WG_TOKENS;
        for (int ks = 0; ks < num_k; ++ks, ++it) {
          const int s = it % WG_STAGES;
          ok = mbar_wait_bounded(&empty_bar[s], ((it / WG_STAGES) & 1) ^ 1, abort_flag);
          if (!ok) break;
          uint8_t* dst = smem + s * WG_STAGE;
          // the leader's barrier counts the bytes of both CTAs
          if (leader) mbar_arrive_expect_tx(&full_bar[s], 2 * WG_STAGE);
          const uint32_t bar = mapa_u32(smem_u32(&full_bar[s]), 0);
          tma_load_2d_pair(dst, &tmap_w, bar, ks * WG_BK, f0);
          tma_load_2d_pair(dst + WG_OPERAND, &tmap_g, bar, ks * WG_BK, b0 + (int)cta_rank * 128);
          if (ks == num_k - 1) {  // this tile's part of S: wanted when its MMAs are done, and the previous tile's has mostly been read by now
            for (int c = 0; c < 4 && ok; ++c) {
              ok = mbar_wait_bounded(&s_empty[c], (lt & 1) ^ 1, abort_flag);
              if (!ok) break;
              mbar_arrive_expect_tx(&s_full[c], WG_S_CHUNK);
              tma_load_2d(smem + WG_S_OFF + c * WG_S_CHUNK, &tmap_s, &s_full[c], f0 + (c & 1) * 64, b0 + (c >> 1) * 128);
            }
            if (!ok) break;
          }
        }
      }
      if (!ok) {
        report_status(p.status, kTimeoutEmptyBarrier, (int)it);
        *abort_flag = 1;
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer (the pair's leader)
    if (leader && elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(256, WG_TOKENS);
      uint32_t it = 0, lt = 0;
      bool ok = true;
      for (long long t = pair; t < n_tiles && ok; t += n_pairs, ++lt) {
        const uint32_t buf = lt & 1;
        ok = mbar_wait_bounded(&acc_empty[buf], ((lt >> 1) & 1) ^ 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        for (int ks = 0; ks < num_k; ++ks, ++it) {
          const int s = it % WG_STAGES;
          ok = mbar_wait_bounded(&full_bar[s], (it / WG_STAGES) & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + s * WG_STAGE);
          const uint64_t a_desc = make_sw128_kmajor_desc(a_addr), b_desc = make_sw128_kmajor_desc(a_addr + WG_OPERAND);
#pragma unroll
          for (int kk = 0; kk < WG_BK / 16; ++kk)
            umma_bf16_ss_pair(tmem_base + buf * WG_TOKENS, a_desc + (uint64_t)(kk * 2), b_desc + (uint64_t)(kk * 2), idesc, (ks > 0 || kk > 0) ? 1u : 0u);
          umma_commit_pair(&empty_bar[s], 3);
        }
        if (ok) umma_commit_pair(&acc_full[buf], 3);
      }
      if (!ok) {
        report_status(p.status, kTimeoutFullBarrier, (int)it);
        *abort_flag = 1;
      }
    }
  } else if (warp >= 4) {
    // ------------------------------------------------------------------ epilogue
    const int q = (warp - 4) & 3, half = (warp - 4) >> 2;  // TMEM lane quarter (32 features), tokens half * 128 .. + 127
    const int fi = (q & 1) * 32 + lane;                    // feature within its chunk of S
    const int chunk = half * 2 + (q >> 1);
    const uint32_t s_base = smem_u32(smem + WG_S_OFF + chunk * WG_S_CHUNK) + (uint32_t)((fi & 7) * 2);
    uint32_t s_off[8];  // a token's row is 128 bytes, its 16-byte pieces permuted by the row index (the loads' swizzle)
#pragma unroll
    for (int i = 0; i < 8; ++i) s_off[i] = s_base + (uint32_t)(((fi >> 3) ^ i) << 4);
    const float half_w = 0.5f * p.window;
    float next_n = 0.0f, next_th = 0.0f;  // of the next tile's feature (past the end: S and the product are zero there, nothing is inside)
    auto feature = [&](long long t) { return (int)(t / token_tiles) * 256 + (int)cta_rank * 128 + q * 32 + lane; };
    auto fetch = [&](long long t) {
      const int f = t < n_tiles ? feature(t) : p.F;
      next_n = f < p.F ? __ldg(p.norm + f) : 0.0f;
      next_th = f < p.F ? __ldg(p.theta + f) : 0.0f;
    };
    fetch(pair);
    uint32_t lt = 0;
    bool ok = true;
    for (long long t = pair; t < n_tiles && ok; t += n_pairs, ++lt) {
      const int f = feature(t);
      const float nf = next_n, th = next_th;
      fetch(t + n_pairs);
      const uint32_t buf = lt & 1;
      ok = __all_sync(0xffffffffu, mbar_wait_bounded(&s_full[chunk], lt & 1, abort_flag) &&
                                       mbar_wait_bounded(&acc_full[buf], (lt >> 1) & 1, abort_flag));
      if (!ok) break;
      tc_fence_after();
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + buf * WG_TOKENS + (uint32_t)(half * 128);
      float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
      int n_in = 0;
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(taddr + (uint32_t)(c * 32), r);
        float s[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          unsigned short u;
          asm volatile("ld.shared.u16 %0, [%1];" : "=h"(u) : "r"(s_off[j & 7] + (uint32_t)((c * 32 + j) * 128)) : "memory");
          s[j] = __uint_as_float((uint32_t)u << 16);
        }
        tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          const float x = s[j] * nf;
          if (x > 0.0f && fabsf(x - th) < half_w) {  // (tokens past the end: S is filled with zeros)
            part[j & 3] += __uint_as_float(r[j]);
            ++n_in;
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&s_empty[chunk]);
        mbar_arrive_cluster(mapa_u32(smem_u32(&acc_empty[buf]), 0));
      }
      if (n_in != 0)
        atomicAdd(p.dtheta + f, (((part[0] + part[1]) + (part[2] + part[3])) / nf + p.add_per_hit * (float)n_in) * (-th / p.window));
    }
    if (!ok) {
      if (lane == 0) report_status(p.status, kTimeoutTmemFull, (int)lt);
      *abort_flag = 1;
    }
  }

  tc_fence_before();
  __syncthreads();
  if (*abort_flag != 0) {
    for (int i = 0; i < 200; ++i) __nanosleep(1000);  // copies that may still be in flight land first
    __syncthreads();
  }
  cluster_sync_all();  // neither CTA may free TMEM or leave while the other can still touch its barriers, shared memory or accumulators
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

int window_grad_gemm_launch(const CUtensorMap& tw, const CUtensorMap& tg, const CUtensorMap& ts, const WindowGradParams& p, cudaStream_t stream) {
  if (p.B <= 0 || p.F <= 0 || p.d <= 0 || p.F % 8 != 0 || p.d % 8 != 0) return (int)cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(window_grad_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, WG_SMEM);
  if (e != cudaSuccess) return (int)e;
  const long long tiles = (long long)((p.F + 255) / 256) * ((p.B + WG_TOKENS - 1) / WG_TOKENS);
  const int pairs = (int)(tiles < 74 ? tiles : 74);
  launch(window_grad_gemm_kernel, 2 * pairs, WG_THREADS, WG_SMEM, stream, tw, tg, ts, p);
  return (int)cudaGetLastError();
}

}  // namespace lmsae
