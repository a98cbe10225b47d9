// fp32 products on the bf16 tensor cores:  C[m, n] = sum_k A[m, k] * B[n, k],  A, B and C fp32, rows of A and B along k (sm_100a).
//
// Each operand is split exactly into three bf16 parts (high, middle, low: 8 bits each, 24 in all), and the six products whose
// weight is above 2^-24 of the result are accumulated: l.h, h.l, m.m, m.h, h.m, h.h, smallest first. The tensor cores cut
// off what does not fit their fp32 accumulator where the fp32 pipes round; over a long sum that is a bias (6e-7 of the result
// at K 768, against an error of 4.6e-7 of the fp32 pipes), so an accumulator holds a slice of 128 of k only and the slices
// are added up, rounded, in registers. Relative error of the 32 largest of 2048 sums, against 64 bits, this and the fp32 pipes:
//   K 64: 0.8e-7 and 1.3e-7; 256: 1.2e-7 and 2.5e-7; 768: 1.2e-7 and 4.3e-7; 2048: 1.3e-7 and 7.1e-7
// Bound by the tensor cores, six times the operations of one bf16 product: 4096 x 24576 x 768: 2505 us (library, fp32 pipes) -> 632 us
// and 37 us for the split. Values that bf16 cannot hold (infinities, NaN, beyond 2^127) mark their row of A or B, and what marked
// rows take part in is redone on the fp32 pipes. So is everything where a wait of the product ran out: it reports to a status word of its
// own call, which no other kernel looks at, and the result is as good as ever.
//
// Structure: CTA pairs (cta_group::2, 256 x 256 tiles) as in encoder_gemm.cu; a tile passes through the accumulator buffers once per
// slice. 384 threads: TMA producer, MMA issuer, TMEM owner, and eight epilogue warps that hold 128 columns of a row each.
//
// LOWER ENDS (ENDS = true), for the TopK encoder, which only needs to know what may be selected (topk_merge.cu): two parts an operand and
// three products (m.h, h.m, h.h), and instead of the estimate h the epilogue stores a lower end of the activation
//     lo = (h - e + bias) * gate,   e = rel * xn * wn >= the error of h   (xn, wn the rows' 2-norms, rel: estimate_rel)
// rounded down to bf16, NaN where the bound says nothing. Bias, gate and rounding are monotone, so that lo encloses the activation of the
// sum in order wherever that is positive; the upper end is at most lo + 2^-7 |lo| + 2 e gate. What a column has of its own comes through shared
// memory, a tile ahead; read from global memory where it was used it kept the epilogue at 13000 cycles a tile, twice what one product takes.
//
// ONE TERM: the first proposal of the TopK encoder. One fp16 part an operand (half_rows_kernel), every row scaled to the top of fp16's range, and what
// rounding took of a row measured and not bounded: 1.9e-4 of its norm as a rule, 4.9e-4 at most. The bound is five times as wide as with two
// bf16 parts at a third of the operations. The largest end of every 32 columns goes along, so that the selection need not read the ends.
// 4096 x 24576 x 768: two parts and three products 24 + 7 + 315 us -> 28 + 165 us. Bound by the epilogue (201 MB of ends), the MMAs take 92.
#include <cuda_fp16.h>
#include "fp32_exact.cuh"
#include "kernels.h"

namespace lmsae {

namespace {

constexpr int FG_BM = 128, FG_BN = 256, FG_BK = 64, FG_STAGES = 6, FG_THREADS = 384;
constexpr int FG_SLICE = 2;  // K blocks of 64 per slice
constexpr int FG_HALF_BYTES = 128 * FG_BK * 2;
constexpr int FG_STAGE_BYTES = 2 * FG_HALF_BYTES;  // this CTA's 128 rows of A and 128 of the 256 rows of B
constexpr int FG_BAR_OFF = FG_STAGES * FG_STAGE_BYTES;
constexpr int FG_STORE_OFF = (FG_BAR_OFF + (2 * FG_STAGES + 4) * 8 + 8 + 15) / 16 * 16;  // ENDS: 32 rows x 32 columns on their way to whole sectors, per epilogue warp
constexpr int FG_COL_OFF = FG_STORE_OFF + 8 * 2048;  // ENDS: what the tile's 256 columns have of their own, for two tiles in turn
constexpr int FG_SMEM = FG_COL_OFF + 2 * 256 * 16 + 1024;

__device__ __forceinline__ void tmem_ld_32x32b_x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
        "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// part of A / B (0 high, 1 middle, 2 low) of the t-th product
template <int TERMS>
__device__ __forceinline__ int part_a(int t) { return TERMS == 1 ? 0 : TERMS == 6 ? (0x201100 >> (4 * (5 - t))) & 15 : t == 0; }
template <int TERMS>
__device__ __forceinline__ int part_b(int t) { return TERMS == 1 ? 0 : TERMS == 6 ? (0x021010 >> (4 * (5 - t))) & 15 : t == 1; }

// dst [rows][PARTS][kp] bf16 = the parts of src [rows][K], zeros behind K; flags[1 + r] = 1 and zeros where a value does not fit, and
// then flags[0] != 0. For lower ends, all optional: norm[r], at least the row's 2-norm and at most 10 % above it; wide[r], at least
// norm[r] * gate[r]; top[0], at least that of every row whose norm is finite; top[1] != 0 where a gate is 0 or NaN. The norm (and the
// width) is infinite where the row's largest magnitude is outside [2^-40, 2^30), bias[r] beyond 2^75 or gate[r] negative, NaN or beyond 2^50: products, (sum + bias) * gate and the
// parts of what is within stay clear of the ends of the fp32 range (2^30 * 2^30 * K 2^14, doubled, * 2^50 < 2^127).
struct SplitBounds {
  float* norm;
  uint16_t* wide;  // bf16
  uint32_t* top;
  const float* bias;
  const float* gate;
};
template <int PARTS>
__global__ void __launch_bounds__(256)
split_bf16_kernel(const float* __restrict__ src, int rows, int K, int kp, __nv_bfloat16* __restrict__ dst, int* __restrict__ flags,
                  const SplitBounds b, const int* wide, int wide_limit) {
  pdl_wait();
  if (wide != nullptr && wide[0] <= wide_limit) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float most = 0.0f;
  for (int r = blockIdx.x * 8 + warp; r < rows; r += gridDim.x * 8) {
    const float* s = src + (size_t)r * K;
    __nv_bfloat16* o = dst + (size_t)r * PARTS * kp;
    bool bad = false;
    unsigned top = 0u;
    float sq = 0.0f;
    for (int c = lane * 4; c < kp; c += 128) {  // (K % 4 == 0, kp % 64 == 0)
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < K) v = __ldg(reinterpret_cast<const float4*>(s + c));
      float x[4] = {v.x, v.y, v.z, v.w}, p[3][4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const unsigned mag = __float_as_uint(x[i]) & 0x7fffffffu;
        top = max(top, mag);
        sq = fmaf(x[i], x[i], sq);
        if (mag >= 0x7f000000u) { bad = true; x[i] = 0.0f; }
        p[0][i] = __bfloat162float(__float2bfloat16(x[i]));
        const float r1 = x[i] - p[0][i];
        p[1][i] = __bfloat162float(__float2bfloat16(r1));
        p[2][i] = r1 - p[1][i];
      }
#pragma unroll
      for (int q = 0; q < PARTS; ++q)
        *reinterpret_cast<uint2*>(o + q * kp + c) = make_uint2(pack_bf16x2(p[q][0], p[q][1]), pack_bf16x2(p[q][2], p[q][3]));
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0 && flags != nullptr) {
      flags[1 + r] = bad ? 1 : 0;
      if (bad) flags[0] = 1;
    }
    if (b.norm != nullptr) {
      top = __reduce_max_sync(0xffffffffu, top);
      sq = warp_sum(sq);
      if (lane == 0) {
        const float gate = b.gate != nullptr ? b.gate[r] : 1.0f;
        bool fits = top == 0u || (top >= 0x2b800000u && top < 0x4e800000u);  // 2^-40, 2^30
        if (b.bias != nullptr) fits &= (__float_as_uint(b.bias[r]) & 0x7fffffffu) < 0x65000000u;  // 2^75
        const bool plain = __float_as_uint(gate) < 0x58800000u;  // 2^50 (and no sign)
        const float n = !(fits && plain) ? __uint_as_float(0x7f800000u) : top == 0u ? 0.0f : 1.05f * sqrtf(sq);
        b.norm[r] = n;
        const float w = mul_up(n, gate);
        if (fits && plain) most = fmaxf(most, w);
        if (b.wide != nullptr) b.wide[r] = fits && plain ? (uint16_t)((__float_as_uint(w) + 0xffffu) >> 16) : (uint16_t)0x7f80u;
        const unsigned gb = __float_as_uint(gate) & 0x7fffffffu;
        if (b.top != nullptr && (gb == 0u || gb > 0x7f800000u)) b.top[1] = 1u;
      }
    }
  }
  if (b.top != nullptr && lane == 0 && most > 0.0f) atomicMax(b.top, __float_as_uint(most));
}

// One fp16 part of the rows of A and of B, scaled by the power of two that brings a row's largest magnitude to [2^14, 2^15):
// dst [rows][kp], zeros behind K, scale[r] the factor that undoes it. What is below 2^-14 then is dropped. norm, wide, top as above (norm at
// most 0.2 % above the 2-norm); a row whose norm is infinite is zeros. lost: at least the 2-norm of what rounding took over that of the row, of
// every row of A, and bits of the largest of all rows of B in top[2].
struct HalfRows {
  const float* src;
  int rows;
  __half* dst;
  float *norm, *scale, *lost;
};
// HELD: rows of at most 1024 stay in registers between the two passes over them (4096 + 24576 rows of 768: 36 -> 28 us).
template <bool HELD>
__global__ void __launch_bounds__(256)
half_rows_kernel(const HalfRows a, const HalfRows b, int K, int kp, const SplitBounds bounds) {
  pdl_wait();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float most = 0.0f, most_lost = 0.0f;
  for (int i = blockIdx.x * 8 + warp; i < a.rows + b.rows; i += gridDim.x * 8) {
    const bool is_b = i >= a.rows;
    const HalfRows& m = is_b ? b : a;
    const int r = is_b ? i - a.rows : i;
    const float* s = m.src + (size_t)r * K;
    unsigned top = 0u;
    float sq = 0.0f;
    float4 held[HELD ? 8 : 1];
    auto look = [&](const float4& v) {
      const float x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        top = max(top, __float_as_uint(x[j]) & 0x7fffffffu);
        sq = fmaf(x[j], x[j], sq);
      }
    };
    if constexpr (HELD) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int c = q * 128 + lane * 4;
        held[q] = c < K ? __ldg(reinterpret_cast<const float4*>(s + c)) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) look(held[q]);
    } else {
      for (int c = lane * 4; c < K; c += 128) look(__ldg(reinterpret_cast<const float4*>(s + c)));
    }
    top = __reduce_max_sync(0xffffffffu, top);
    sq = warp_sum(sq);
    bool fits = top == 0u || (top >= 0x2b800000u && top < 0x4e800000u);  // 2^-40, 2^30
    const float gate = is_b && bounds.gate != nullptr ? bounds.gate[r] : 1.0f;
    if (is_b && bounds.bias != nullptr) fits &= (__float_as_uint(bounds.bias[r]) & 0x7fffffffu) < 0x65000000u;  // 2^75
    fits &= __float_as_uint(gate) < 0x58800000u;  // 2^50 (and no sign)
    const int shift = fits && top != 0u ? 14 + 127 - (int)(top >> 23) : 0;
    const float up = __uint_as_float((unsigned)(127 + shift) << 23);
    if (lane == 0) {
      const float n = !fits ? __uint_as_float(0x7f800000u) : top == 0u ? 0.0f : 1.001f * sqrtf(sq);
      m.norm[r] = n;
      m.scale[r] = __uint_as_float((unsigned)(127 - shift) << 23);
      if (is_b) {
        const float w = mul_up(n, gate);
        if (fits) most = fmaxf(most, w);
        bounds.wide[r] = fits ? (uint16_t)((__float_as_uint(w) + 0xffffu) >> 16) : (uint16_t)0x7f80u;
        const unsigned gb = __float_as_uint(gate) & 0x7fffffffu;
        if (gb == 0u || gb > 0x7f800000u) bounds.top[1] = 1u;
      }
    }
    __half* o = m.dst + (size_t)r * kp;
    float all = 0.0f, gone = 0.0f;
    auto convert = [&](int c, float4 v) {
      if (!fits) v = make_float4(0.f, 0.f, 0.f, 0.f);
      float x[4] = {v.x * up, v.y * up, v.z * up, v.w * up};
      __half y[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        y[j] = __float2half_rn(fabsf(x[j]) < 6.103515625e-5f ? 0.0f : x[j]);  // 2^-14: no fp16 subnormals
        const float rest = x[j] - __half2float(y[j]);
        all = fmaf(x[j], x[j], all);
        gone = fmaf(rest, rest, gone);
      }
      const __half2 lo = __halves2half2(y[0], y[1]), hi = __halves2half2(y[2], y[3]);
      *reinterpret_cast<uint2*>(o + c) = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
    };
    if constexpr (HELD) {
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q * 128 + lane * 4 < kp) convert(q * 128 + lane * 4, held[q]);
    } else {
      for (int c = lane * 4; c < kp; c += 128) convert(c, c < K ? __ldg(reinterpret_cast<const float4*>(s + c)) : make_float4(0.f, 0.f, 0.f, 0.f));
    }
    all = warp_sum(all);
    gone = warp_sum(gone);
    if (lane == 0) {
      const float lost = all > 0.0f ? 1.002f * sqrtf(gone / all) : 0.0f;
      if (is_b) most_lost = fmaxf(most_lost, lost);
      else m.lost[r] = lost;
    }
  }
  if (lane == 0 && most_lost > 0.0f) atomicMax(bounds.top + 2, __float_as_uint(most_lost));
  if (lane == 0 && most > 0.0f) atomicMax(bounds.top, __float_as_uint(most));
}

struct Fp32GemmParams {
  int M, N, kp;
  long long ldc;
  int m_tiles, n_tiles, pairs;
  float* C;            // [M][ldc], or the lower ends
  __nv_bfloat16* lo;
  float rel;           // ENDS: the bound's factor, the rows' norms, and the columns' bias and gate (nullptr: 0 and 1)
  const float* na;
  const float* nb;
  const float* bias;
  const float* gate;
  const float* sa;     // one term: what a row of A and of B was divided by
  const float* sb;
  const float* lost;   // one term: what rounding took of a row of A, and the most that it took of one of B
  const uint32_t* lost_b;
  const int* wide;     // optional: nothing is done unless wide[0] > wide_limit
  int wide_limit;
  float* maxima;       // one term: [M][ld_maxima], the largest end of every 32 columns (group_max)
  long long ld_maxima;
  int* status;
};

// The largest end of a group of columns, none below 0, rounded down to bf16; the last bit is set where an end says nothing.
__device__ __forceinline__ float group_max(float top, bool unknown) {
  const uint32_t b = __float_as_uint(top);
  return __uint_as_float((b >= 0x7f800000u ? 0u : b & 0xffff0000u) | (unknown ? 1u : 0u));
}

template <int TERMS, bool ENDS>
__global__ void __launch_bounds__(FG_THREADS, 1)
fp32_gemm_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b, const Fp32GemmParams p) {
  pdl_wait();
  if (p.wide != nullptr && p.wide[0] <= p.wide_limit) return;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + FG_BAR_OFF);
  uint64_t* empty_bar = full_bar + FG_STAGES;
  uint64_t* tmem_full_bar = empty_bar + FG_STAGES;
  uint64_t* tmem_empty_bar = tmem_full_bar + 2;
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(tmem_empty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();
  const bool leader = cta_rank == 0;
  const int pair = (int)(blockIdx.x >> 1);
  const int tiles = p.m_tiles * p.n_tiles, k_blocks = p.kp / FG_BK;
  const int slice = ENDS ? k_blocks : FG_SLICE, slices = (k_blocks + slice - 1) / slice;  // (a lower end needs no slices: estimate_rel)

  if (threadIdx.x == 0) {
    for (int i = 0; i < FG_STAGES; ++i) {
      mbar_init(&full_bar[i], 1);
      mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&tmem_full_bar[i], 1);
      mbar_init(&tmem_empty_bar[i], 16);  // the epilogue warps of both CTAs
    }
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 0 && lane == 0) {
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&tmap_b);
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
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      for (int t = pair; t < tiles && ok; t += p.pairs) {
        // (pairs that run together work on neighbouring row panels of the same columns)
        const int m0 = (t % p.m_tiles) * 2 * FG_BM + (int)cta_rank * FG_BM, n0 = (t / p.m_tiles) * FG_BN + (int)cta_rank * FG_BM;
        for (int kb0 = 0; kb0 < k_blocks && ok; kb0 += slice) {
          const int n_kb = min(slice, k_blocks - kb0);
          for (int j = 0; j < TERMS * n_kb; ++j, ++it) {
            const int term = j / n_kb, kx = (kb0 + j % n_kb) * FG_BK;
            const int s = it % FG_STAGES;
            if (!mbar_wait_bounded(&empty_bar[s], ((it / FG_STAGES) & 1) ^ 1, abort_flag)) {
              report_status(p.status, kTimeoutEmptyBarrier, (int)it);
              *abort_flag = 1;
              ok = false;
              break;
            }
            uint8_t* dst = smem + s * FG_STAGE_BYTES;
            if (leader) mbar_arrive_expect_tx(&full_bar[s], 2 * FG_STAGE_BYTES);
            const uint32_t bar = mapa_u32(smem_u32(&full_bar[s]), 0);
            tma_load_2d_pair(dst, &tmap_a, bar, part_a<TERMS>(term) * p.kp + kx, m0);
            tma_load_2d_pair(dst + FG_HALF_BYTES, &tmap_b, bar, part_b<TERMS>(term) * p.kp + kx, n0);
          }
        }
      }
    }
  } else if (warp == 1) {
    if (leader && elect_one()) {
      constexpr uint32_t idesc = TERMS == 1 ? make_idesc_f16(2 * FG_BM, FG_BN) : make_idesc_bf16(2 * FG_BM, FG_BN);
      uint32_t it = 0, sub = 0;
      bool ok = true;
      for (int t = pair; t < tiles && ok; t += p.pairs) {
        for (int kb0 = 0; kb0 < k_blocks && ok; kb0 += slice, ++sub) {
          const int buf = sub & 1;
          if (!mbar_wait_bounded(&tmem_empty_bar[buf], ((sub >> 1) & 1) ^ 1, abort_flag)) {
            report_status(p.status, kTimeoutTmemEmpty, (int)sub);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t tmem_d = tmem_base + (uint32_t)(buf * FG_BN);
          const int steps = TERMS * min(slice, k_blocks - kb0);
          for (int j = 0; j < steps; ++j, ++it) {
            const int s = it % FG_STAGES;
            if (!mbar_wait_bounded(&full_bar[s], (it / FG_STAGES) & 1, abort_flag)) {
              report_status(p.status, kTimeoutFullBarrier, (int)it);
              *abort_flag = 1;
              ok = false;
              break;
            }
            tc_fence_after();
            const uint32_t a_addr = smem_u32(smem + s * FG_STAGE_BYTES);
            const uint64_t a_desc = make_sw128_kmajor_desc(a_addr), b_desc = make_sw128_kmajor_desc(a_addr + FG_HALF_BYTES);
#pragma unroll
            for (int kk = 0; kk < FG_BK / 16; ++kk)
              umma_bf16_ss_pair(tmem_d, a_desc + (uint64_t)(kk * 2), b_desc + (uint64_t)(kk * 2), idesc, (j > 0 || kk > 0) ? 1u : 0u);
            umma_commit_pair(&empty_bar[s], 3);
          }
          if (ok) umma_commit_pair(&tmem_full_bar[buf], 3);
        }
      }
    }
  } else if (warp >= 4) {
    const int q = warp & 3, half = (warp - 4) >> 2;  // TMEM lane quarter, column half
    const bool vec = ENDS ? p.N % 8 == 0 && p.ldc % 8 == 0 && (reinterpret_cast<uintptr_t>(p.lo) & 15) == 0
                          : p.N % 4 == 0 && p.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(p.C) & 15) == 0;
    uint32_t sub = 0;
    bool ok = true;
    // what column threadIdx.x - 128 of tile t has of its own: scale, norm, bias, gate
    auto column = [&](int t) -> float4 {
      const int c = (t / p.m_tiles) * FG_BN + (int)threadIdx.x - 128;
      float4 v = make_float4(1.0f, 0.0f, 0.0f, 1.0f);
      if (t < tiles && c < p.N) {
        if (TERMS == 1) v.x = __ldg(p.sb + c);
        v.y = __ldg(p.nb + c);
        if (p.bias != nullptr) v.z = __ldg(p.bias + c);
        if (p.gate != nullptr) v.w = __ldg(p.gate + c);
      }
      return v;
    };
    float4 ahead = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if constexpr (ENDS) ahead = column(pair);
    for (int t = pair; t < tiles && (ENDS || ok); t += p.pairs) {
      const int row = (t % p.m_tiles) * 2 * FG_BM + (int)cta_rank * FG_BM + q * 32 + lane;
      const int c0 = (t / p.m_tiles) * FG_BN + half * 128;
      if constexpr (ENDS) {
        // (a warp that gave up goes on to the barriers, which the others wait at without a limit)
        float4* cols = reinterpret_cast<float4*>(smem + FG_COL_OFF) + (sub & 1) * 256;
        cols[threadIdx.x - 128] = ahead;
        asm volatile("bar.sync 1, 256;" ::: "memory");
        ahead = column(t + p.pairs);
        const int buf = sub & 1;
        ++sub;
        if (ok && !__all_sync(0xffffffffu, mbar_wait_bounded(&tmem_full_bar[buf], ((sub - 1) >> 1) & 1, abort_flag))) {
          if (lane == 0) report_status(p.status, kTimeoutTmemFull, (int)sub);
          *abort_flag = 1;
          ok = false;
        }
        if (!ok) continue;
        tc_fence_after();
        const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * FG_BN + half * 128);
        const int row0 = row - lane;
        const float rx = row < p.M ? -mul_up(TERMS == 1 ? half_rel(p.rel, __ldg(p.lost + row), p.lost_b) : p.rel, __ldg(p.na + row)) : 0.0f;
        const float sr = TERMS == 1 && row < p.M ? __ldg(p.sa + row) : 1.0f;
        uint8_t* tile_s = smem + FG_STORE_OFF + (warp - 4) * 2048;
        float largest[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t r[32];
          tmem_ld_32x32b_x32(taddr + (uint32_t)(g * 32), r);
          tmem_wait_ld();
          if (g == 3) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&tmem_empty_bar[buf]), 0));
          }
          const int cg = c0 + g * 32;
          float top = 0.0f;
          bool unknown = false;
          uint4 o[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint32_t e[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float4 c = cols[half * 128 + g * 32 + j * 8 + i];  // (the same for the whole warp)
              float v = __uint_as_float(r[j * 8 + i]);
              if constexpr (TERMS == 1) v = mul_rn(v, sr * c.x);  // (powers of two)
              v = mul_rn(add_rn(fma_rn(rx, c.y, v), c.z), c.w);
              const uint32_t b = __float_as_uint(v);
              const bool none = (b & 0x7f800000u) == 0x7f800000u;
              e[i] = none ? 0x7fffu : ((int)b < 0 ? b + 0xffffu : b) >> 16;  // rounded down
              unknown |= none;
              top = fmaxf(top, v);
            }
            o[j] = make_uint4(e[0] | e[1] << 16, e[2] | e[3] << 16, e[4] | e[5] << 16, e[6] | e[7] << 16);
          }
          largest[g] = group_max(top, unknown);
          // through shared memory, so that four lanes write whole sectors of a row (as in encoder_gemm.cu)
          __syncwarp();
#pragma unroll
          for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(tile_s + lane * 64 + ((j ^ ((lane >> 1) & 3)) * 16)) = o[j];
          __syncwarp();
          if (vec) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int rr = i * 8 + (lane >> 2), j = lane & 3;
              const uint4 v = *reinterpret_cast<const uint4*>(tile_s + rr * 64 + ((j ^ ((rr >> 1) & 3)) * 16));
              if (row0 + rr < p.M && cg + j * 8 < p.N) *reinterpret_cast<uint4*>(p.lo + (row0 + rr) * p.ldc + cg + j * 8) = v;
            }
          } else {  // lane: a column
            for (int rr = 0; rr < 32; ++rr) {
              const int j = lane >> 3;
              const unsigned short v = *reinterpret_cast<const unsigned short*>(tile_s + rr * 64 + ((j ^ ((rr >> 1) & 3)) * 16) + (lane & 7) * 2);
              if (row0 + rr < p.M && cg + lane < p.N) reinterpret_cast<unsigned short*>(p.lo)[(row0 + rr) * p.ldc + cg + lane] = v;
            }
          }
        }
        if (p.maxima != nullptr && row < p.M)
          *reinterpret_cast<float4*>(p.maxima + row * p.ld_maxima + c0 / 32) = make_float4(largest[0], largest[1], largest[2], largest[3]);
      } else {
        float acc[128];
#pragma unroll
        for (int j = 0; j < 128; ++j) acc[j] = 0.0f;
        for (int s = 0; s < slices; ++s, ++sub) {
          const int buf = sub & 1;
          if (!__all_sync(0xffffffffu, mbar_wait_bounded(&tmem_full_bar[buf], (sub >> 1) & 1, abort_flag))) {
            if (lane == 0) report_status(p.status, kTimeoutTmemFull, (int)sub);
            *abort_flag = 1;
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * FG_BN + half * 128);
#pragma unroll
          for (int g = 0; g < 8; ++g) {
            uint32_t r[16];
            tmem_ld_32x32b_x16(taddr + (uint32_t)(g * 16), r);
            tmem_wait_ld();
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[g * 16 + j] += __uint_as_float(r[j]);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(mapa_u32(smem_u32(&tmem_empty_bar[buf]), 0));
        }
        if (ok && row < p.M) {
          float* dst = p.C + row * p.ldc + c0;
          if (vec) {
#pragma unroll
            for (int j = 0; j < 128; j += 4)
              if (c0 + j < p.N) *reinterpret_cast<float4*>(dst + j) = make_float4(acc[j], acc[j + 1], acc[j + 2], acc[j + 3]);
          } else {
#pragma unroll
            for (int j = 0; j < 128; ++j)
              if (c0 + j < p.N) dst[j] = acc[j];
          }
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
  cluster_sync_all();  // neither CTA may free TMEM or leave while the other can still touch its barriers or accumulators
  if (warp == 2) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// C[m, n] of marked rows of A or of B on the fp32 pipes, a warp per element; leaves at once where nothing is marked.
__global__ void __launch_bounds__(256)
marked_products_kernel(const float* __restrict__ A, const float* __restrict__ B, int M, int N, int K, const int* __restrict__ fa,
                       const int* __restrict__ fb, float* __restrict__ C, long long ldc, const int* __restrict__ status) {
  pdl_wait();
  const bool all = status[0] != 0;
  if (fa[0] == 0 && fb[0] == 0 && !all) return;
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * 8;
  for (long long e = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); e < (long long)M * N; e += warps) {
    const int m = (int)(e / N), n = (int)(e - (long long)m * N);
    if (!all && fa[1 + m] == 0 && fb[1 + n] == 0) continue;
    float s = 0.0f;
    for (int k = lane; k < K; k += 32) s = fmaf(A[(size_t)m * K + k], B[(size_t)n * K + k], s);
    s = warp_sum(s);
    if (lane == 0) C[m * ldc + n] = s;
  }
}

}  // namespace

int split_bf16_launch(const float* src, int rows, int K, int kp, int parts, __nv_bfloat16* dst, int* flags, float* norm, uint16_t* wide, uint32_t* top,
                      const float* bias, const float* gate, cudaStream_t stream) {
  if (K % 4 != 0 || kp % 64 != 0 || kp < K || (reinterpret_cast<uintptr_t>(src) & 15) != 0 || (parts != 2 && parts != 3)) return (int)cudaErrorInvalidValue;
  const int blocks = (rows + 7) / 8;
  auto kern = parts == 2 ? split_bf16_kernel<2> : split_bf16_kernel<3>;
  launch(kern, blocks < 148 * 8 ? blocks : 148 * 8, 256, 0, stream, src, rows, K, kp, dst, flags, SplitBounds{norm, wide, top, bias, gate}, nullptr, 0);
  return (int)cudaGetLastError();
}

static cudaError_t launch_product(const void* kernel, const CUtensorMap& ta, const CUtensorMap& tb, Fp32GemmParams& p, cudaStream_t stream) {
  p.m_tiles = (p.M + 2 * FG_BM - 1) / (2 * FG_BM);
  p.n_tiles = (p.N + FG_BN - 1) / FG_BN;
  const long long tiles = (long long)p.m_tiles * p.n_tiles;
  if (tiles > 2147483647LL - 148) return cudaErrorInvalidValue;
  p.pairs = (int)(tiles < 74 ? tiles : 74);
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FG_SMEM);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * p.pairs);
  cfg.blockDim = dim3(FG_THREADS);
  cfg.dynamicSmemBytes = FG_SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  void* args[3] = {const_cast<CUtensorMap*>(&ta), const_cast<CUtensorMap*>(&tb), &p};
  ++kernel_launches;
  return cudaLaunchKernelExC(&cfg, kernel, args);
}

int fp32_gemm_launch(const CUtensorMap& ta, const CUtensorMap& tb, const float* A, const float* B, int M, int N, int K, int kp, const int* fa,
                     const int* fb, float* C, long long ldc, int* status, bool tensor_cores, cudaStream_t stream) {
  Fp32GemmParams p = {};
  p.M = M; p.N = N; p.kp = kp; p.C = C; p.ldc = ldc; p.status = status;
  if (tensor_cores) {
    const cudaError_t e = launch_product(reinterpret_cast<const void*>(fp32_gemm_kernel<6, false>), ta, tb, p, stream);
    if (e != cudaSuccess) return (int)e;
  }
  launch(marked_products_kernel, 148 * 8, 256, 0, stream, A, B, M, N, K, fa, fb, C, ldc, status);
  return (int)cudaGetLastError();
}

int fp32_ends_launch(const CUtensorMap& ta, const CUtensorMap& tb, int M, int N, int K, int kp, const float* na, const float* nb, const float* bias,
                     const float* gate, __nv_bfloat16* lo, long long ldc, int* status, const int* wide, int wide_limit, cudaStream_t stream) {
  Fp32GemmParams p = {};
  p.M = M; p.N = N; p.kp = kp; p.lo = lo; p.ldc = ldc; p.status = status; p.wide = wide; p.wide_limit = wide_limit;
  p.rel = estimate_rel(K); p.na = na; p.nb = nb; p.bias = bias; p.gate = gate;
  return (int)launch_product(reinterpret_cast<const void*>(fp32_gemm_kernel<3, true>), ta, tb, p, stream);
}

int half_rows_launch(const float* A, int M, __half* a16, float* na, float* sa, float* lost, const float* B, int N, __half* b16, float* nb, float* sb, int K, int kp,
                     uint16_t* widths, uint32_t* top, const float* bias, const float* gate, cudaStream_t stream) {
  if (K % 4 != 0 || kp % 64 != 0 || kp < K || ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15) != 0) return (int)cudaErrorInvalidValue;
  const long long blocks = ((long long)M + N + 7) / 8;
  auto kern = K <= 1024 ? half_rows_kernel<true> : half_rows_kernel<false>;
  return (int)launch(kern, (int)(blocks < 148 * 8 ? blocks : 148 * 8), 256, 0, stream, HalfRows{A, M, a16, na, sa, lost},
                     HalfRows{B, N, b16, nb, sb, nullptr}, K, kp, SplitBounds{nullptr, widths, top, bias, gate});
}

int half_ends_launch(const CUtensorMap& ta, const CUtensorMap& tb, int M, int N, int K, int kp, const float* na, const float* sa, const float* lost,
                     const uint32_t* top, const float* nb, const float* sb, const float* bias, const float* gate, __nv_bfloat16* lo, long long ldc, float* maxima,
                     long long ld_maxima, int* status, cudaStream_t stream) {
  if (maxima != nullptr && (ld_maxima % 4 != 0 || ld_maxima < (long long)(N + FG_BN - 1) / FG_BN * 8 || (reinterpret_cast<uintptr_t>(maxima) & 15) != 0))
    return (int)cudaErrorInvalidValue;
  Fp32GemmParams p = {};
  p.M = M; p.N = N; p.kp = kp; p.lo = lo; p.ldc = ldc; p.status = status;
  p.maxima = maxima; p.ld_maxima = ld_maxima;
  p.rel = estimate_rel_half(K); p.na = na; p.sa = sa; p.lost = lost; p.lost_b = top + 2; p.nb = nb; p.sb = sb; p.bias = bias; p.gate = gate;
  return (int)launch_product(reinterpret_cast<const void*>(fp32_gemm_kernel<1, true>), ta, tb, p, stream);
}

int split_bf16_if_launch(const float* src, int rows, int K, int kp, __nv_bfloat16* dst, const int* wide, int wide_limit, cudaStream_t stream) {
  if (K % 4 != 0 || kp % 64 != 0 || kp < K || (reinterpret_cast<uintptr_t>(src) & 15) != 0) return (int)cudaErrorInvalidValue;
  const int blocks = (rows + 7) / 8;
  return (int)launch(split_bf16_kernel<2>, blocks < 148 * 8 ? blocks : 148 * 8, 256, 0, stream, src, rows, K, kp, dst, nullptr, SplitBounds{}, wide, wide_limit);
}

}  // namespace lmsae
