// Sparse gradient rows + Adam, streamed row by row (sm_100a): the update of every fused training step.
//
// For a feature row f the gradient rows
//     dW_D[f, :] = sum over its entries of act * d x_hat[token, :]        (decoder side)
//     dW_E^T[f, :] = sum over its entries of dact * x[token, :]           (encoder side)
// are rebuilt in registers from the entry list and Adam is applied in the same pass; with `dact_mode` the decoder side also
// computes the code gradients  dact = d x_hat[token, :] . bf16(W_D[f, :])  it has both factors of in registers, so that no
// kernel gathers the decoder rows a second time for them (a pass over B * k rows: about as much L2 traffic as the decoder's).
//
// What bounds it: 26 bytes of HBM traffic per parameter (p, m, v in fp32 in and out, bf16 shadow out). What kept the
// previous warp-per-row and CTA-per-row forms at 0.6-0.8 of the copy rate is that a row alternated between a gather phase
// (entry list -> codes -> gathered rows, several L2 latencies) and a phase in which its own streams were on their way. Here the
// three streams of a row are fetched by bulk copies into shared memory, issued as soon as the previous row's values
// have been read, i.e. BEFORE the gathers of their row start; values go back with plain streaming stores.
//
//   group of W warps   one feature row at a time; a thread owns four consecutive columns of every chunk of 128 W columns
//   W                  1 up to 1024 columns, 2 up to 2048, 4 up to 4096, 8 up to 8192: at most eight chunks (32 gradient
//                      registers) per thread, and 14 bytes x d of shared memory per group leave four or more groups per SM
//                      up to 4096 columns
//   rows               dealt out in small chunks by a counter (entry counts are skewed: a static deal left SMs idle)
//   long lists         a row with more than kHeavyRow entries (dense features; a few rows of a Lorsa dictionary hold an entry of
//                      EVERY token) is processed by all groups of a CTA, which share its entries and add up their partial
//                      rows; one warp alone took 1.1 ms for 2048 entries (the whole launch: 1167 -> 130 us, 8192 rows of 768). Pieces of the list are
//                      cut so that every group gets the same share: 450 entries in pieces of 32 kept 6 of 20 groups idle and the others
//                      twice as long as 23 each do (a Lorsa step whose 546 long rows hold 245000 of 262144 entries: 737 -> 713 us)
//
// Measured, previous kernels (+ the pass for the code gradients where this one replaces it) -> this one:
//   131072 rows of 4096, both sides          5.09 + 0.43 -> 4.75 ms  (27.9 GB: 5.9 TB/s)
//   12 + 78 matrices of 24576 x 768 (CLT)    8.62 + 3.05 -> 7.59 ms  (44 GB: 5.8 TB/s)
//   24576 rows of 768, both sides, k 50      222 + 155   -> 182 us
//   32768 rows of 2048, both sides, k 128    1103 + 590  -> 819 us (16 entries a row: bound by the gathers, 4.3 GB)
#include "adam.cuh"
#include "gather.cuh"
#include "kernels.h"

namespace lmsae {

LMSAE_DEFINE_BOUNDS_FETCH(bounds_fetch_grad_adam)

namespace {

template <int W>
__device__ __forceinline__ void group_sync(int gid) {
  if constexpr (W == 1) {
    __syncwarp();
  } else {
    asm volatile("bar.sync %0, %1;" ::"r"(gid + 1), "n"(W * 32) : "memory");
  }
}

// Whether all threads of the group say so (a barrier of the group).
template <int W>
__device__ __forceinline__ bool group_all(int gid, bool ok) {
  if constexpr (W == 1) {
    return __all_sync(0xffffffffu, ok);
  } else {
    uint32_t r;
    __syncwarp();
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        "setp.ne.u32 q, %3, 0;\n\t"
        "barrier.cta.red.and.pred p, %1, %2, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}"
        : "=r"(r)
        : "r"(gid + 1), "n"(W * 32), "r"((uint32_t)ok)
        : "memory");
    return r != 0;
  }
}

// Position of a thread in its group and the group's slice of shared memory.
struct GroupCtx {
  int gid, wg, lane, tid;  // group, warp within it, lane, thread within it
  float* stage;            // [3][d]: parameter, first and second moment of the row in flight
  uint2* rounded;          // [NCH * T] bf16-rounded parameters of the row, four columns each
  float* dots;             // [W][32] partial dot products (W > 1)
};

// Entries whose rows are requested at once, as the registers allow: with short rows a feature's time is the latency of its entries' rows, one
// group of them after the other (512 x 8 codes of 256 rows of 64: 29 -> 23 us; four at a time of rows of 512 spilled and gained nothing).
template <int NCH>
__host__ __device__ constexpr int gather_batch() { return NCH == 1 ? 8 : NCH == 2 ? 4 : 2; }

// Rebuilds this group's share of one gradient row: entries [e0 + 32 * first, e1) in batches of 32, every `stride`-th batch.
// g += coefficient * row, with DOT also the code gradients against the bf16-rounded row in c.rounded. Returns (encoder side)
// the sum of this lane's coefficients.
template <bool IS_D, bool DOT, int W, int NCH>
__device__ __forceinline__ float gather_side(const GradAdamParams& p, const GroupCtx& c, const __nv_bfloat16* src, int e0, int e1, int first, int stride, int piece,
                                             float (&g)[NCH][4]) {
  constexpr int Q = gather_batch<NCH>();
  float coef_sum = 0.0f;
  for (int eb = e0 + first * piece; eb < e1; eb += stride * piece) {
    const int n_e = min(piece, e1 - eb);
    int row_l = 0, ent_l = 0;
    float a_l = 0.0f;
    if (c.lane < n_e) {
      ent_l = (int)LMSAE_IDX(p.entries[eb + c.lane], p.n_codes);
      row_l = (int)LMSAE_IDX(ent_l / p.k, p.n_rows);
      a_l = IS_D ? p.act[ent_l] : __ldcg(p.dact + ent_l);
    }
    if (!IS_D) coef_sum += a_l;
    float dot_l = 0.0f;
    unsigned mask = __ballot_sync(0xffffffffu, a_l != 0.0f);  // (the same in every warp of the group)
    while (mask != 0u) {
      // a few entries at a time: all their loads are requested before the first is used
      int j[Q];
      float a[Q];
      uint2 u[Q][NCH];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        j[q] = -1;
        a[q] = 0.0f;
        if (mask != 0u) {
          j[q] = __ffs(mask) - 1;
          mask &= mask - 1u;
          a[q] = __shfl_sync(0xffffffffu, a_l, j[q]);
          const __nv_bfloat16* r = src + (size_t)__shfl_sync(0xffffffffu, row_l, j[q]) * p.d + c.tid * 4;
#pragma unroll
          for (int i = 0; i < NCH; ++i) {
            if (i * W * 128 + c.tid * 4 < p.d) u[q][i] = __ldg(reinterpret_cast<const uint2*>(r + i * W * 128));
            else u[q][i] = make_uint2(0u, 0u);
          }
        } else {
#pragma unroll
          for (int i = 0; i < NCH; ++i) u[q][i] = make_uint2(0u, 0u);
        }
      }
      float d0[Q], d1[Q];
#pragma unroll
      for (int q = 0; q < Q; ++q) d0[q] = d1[q] = 0.0f;
#pragma unroll
      for (int i = 0; i < NCH; ++i) {
        float w0 = 0.f, w1 = 0.f, w2 = 0.f, w3 = 0.f;
        if constexpr (DOT) {
          const uint2 w = c.rounded[i * W * 32 + c.tid];
          w0 = __uint_as_float(w.x << 16); w1 = __uint_as_float(w.x & 0xffff0000u);
          w2 = __uint_as_float(w.y << 16); w3 = __uint_as_float(w.y & 0xffff0000u);
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) {  // (an absent entry adds zeros)
          const float x0 = __uint_as_float(u[q][i].x << 16), x1 = __uint_as_float(u[q][i].x & 0xffff0000u);
          const float x2 = __uint_as_float(u[q][i].y << 16), x3 = __uint_as_float(u[q][i].y & 0xffff0000u);
          fma2(g[i][0], g[i][1], x0, x1, a[q], a[q]);
          fma2(g[i][2], g[i][3], x2, x3, a[q], a[q]);
          if constexpr (DOT) {
            fma2(d0[q], d1[q], x0, x1, w0, w1);
            fma2(d0[q], d1[q], x2, x3, w2, w3);
          }
        }
      }
      if constexpr (DOT) {
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          const float dot = warp_sum(d0[q] + d1[q]);
          if (c.lane == j[q]) dot_l = dot;
        }
      }
    }
    if constexpr (DOT) {
      if constexpr (W > 1) {
        c.dots[c.wg * 32 + c.lane] = dot_l;
        group_sync<W>(c.gid);
        if (c.wg == 0) {
          dot_l = 0.0f;
#pragma unroll
          for (int w = 0; w < W; ++w) dot_l += c.dots[w * 32 + c.lane];
        }
      }
      if (c.wg == 0 && c.lane < n_e) {
        float* o = p.dact_out + ent_l;
        *o = p.dact_mode == 2 ? *o + dot_l : dot_l;
      }
      group_sync<W>(c.gid);  // the partial sums may be overwritten, and the other warps may read the code gradients
    }
  }
  return coef_sum;
}

// The bf16-rounded row the forward pass used (what the shadow holds), from the fp32 row in shared memory. A thread writes and
// later reads its own columns only.
template <int W, int NCH>
__device__ __forceinline__ void round_row(const float* row, int d, const GroupCtx& c) {
#pragma unroll
  for (int i = 0; i < NCH; ++i) {
    const int col = i * W * 128 + c.tid * 4;
    uint2 r = make_uint2(0u, 0u);  // (columns past the end multiply zeros: they must not hold a NaN)
    if (col < d) {
      const float4 w = *reinterpret_cast<const float4*>(row + col);
      r = make_uint2(pack_bf16x2(w.x, w.y), pack_bf16x2(w.z, w.w));
    }
    c.rounded[i * W * 32 + c.tid] = r;
  }
}

// Scales the gradient row, accumulates its squared norm, and applies Adam from the stage. Returns this thread's share of
// the new decoder row's squared norm.
template <bool IS_D, int W, int NCH>
__device__ __forceinline__ float apply_side(const GradAdamParams& p, const GroupCtx& c, int f, float gmul, const AdamConst& h,
                                            float (&g)[NCH][4], float& gsq) {
  float* Wp = IS_D ? p.WD : p.WE;
  float* Mp = IS_D ? p.mD : p.mE;
  float* Vp = IS_D ? p.vD : p.vE;
  __nv_bfloat16* Sp = IS_D ? p.WD_bf16 : p.WE_bf16;
  const size_t o = (size_t)f * p.d, os = (size_t)(f - p.state_f0) * p.d;
  const float self_scale = (IS_D && p.wd_self_scale != nullptr) ? p.wd_self_scale[f] * gmul : 0.0f;
  float norm_sq = 0.0f;
#pragma unroll
  for (int i = 0; i < NCH; ++i) {
    const int col = i * W * 128 + c.tid * 4;
    if (col >= p.d) continue;
#pragma unroll
    for (int q = 0; q < 4; ++q) g[i][q] *= gmul;
    if (p.grad_sq_sum != nullptr) gsq += g[i][0] * g[i][0] + g[i][1] * g[i][1] + g[i][2] * g[i][2] + g[i][3] * g[i][3];
    if (!p.update) continue;
    float4 w = *reinterpret_cast<const float4*>(c.stage + col);
    float4 m = *reinterpret_cast<const float4*>(c.stage + p.d + col);
    float4 v = *reinterpret_cast<const float4*>(c.stage + 2 * p.d + col);
    if (IS_D) {  // (not part of the squared gradient norm: a penalty term's share is small)
      g[i][0] = fmaf(self_scale, w.x, g[i][0]); g[i][1] = fmaf(self_scale, w.y, g[i][1]);
      g[i][2] = fmaf(self_scale, w.z, g[i][2]); g[i][3] = fmaf(self_scale, w.w, g[i][3]);
    }
    adam_update(w.x, m.x, v.x, g[i][0], h); adam_update(w.y, m.y, v.y, g[i][1], h);
    adam_update(w.z, m.z, v.z, g[i][2], h); adam_update(w.w, m.w, v.w, g[i][3], h);
    __stcs(reinterpret_cast<float4*>(Wp + o + col), w);
    __stcs(reinterpret_cast<float4*>(Mp + os + col), m);
    __stcs(reinterpret_cast<float4*>(Vp + os + col), v);
    if (IS_D) norm_sq += w.x * w.x + w.y * w.y + w.z * w.z + w.w * w.w;
    uint2 sh;
    sh.x = pack_bf16x2(w.x, w.y);
    sh.y = pack_bf16x2(w.z, w.w);
    *reinterpret_cast<uint2*>(Sp + o + col) = sh;
  }
  return norm_sq;
}

template <int NCH>
constexpr int rows_threads() { return NCH <= 4 ? 768 : NCH <= 6 ? 640 : 512; }

}  // namespace

template <int W, int NCH>
__global__ void __launch_bounds__(rows_threads<NCH>(), 1)
grad_adam_rows_kernel(const GradAdamParams p) {
  pdl_wait();
  if (p.longest < 0 && !any_longer_list(p, -p.longest)) return;  // (the launch of the other kernel did it)
  constexpr int T = 32 * W;
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const int G = (int)blockDim.x / T;
  GroupCtx c;
  c.gid = (int)threadIdx.x / T;
  c.tid = (int)threadIdx.x % T;
  c.wg = c.tid >> 5;
  c.lane = (int)threadIdx.x & 31;
  float* stages = reinterpret_cast<float*>(smem_raw);
  uint2* rounded = reinterpret_cast<uint2*>(stages + (size_t)G * 3 * p.d);  // [G][NCH * T]
  float* dots = reinterpret_cast<float*>(rounded + (size_t)G * NCH * T);    // [G][W][32]
  float* red = dots + (size_t)G * W * 32;                // [2][G][W] norms, then [G] bias sums
  float* bias_part = red + 2 * G * W;
  uint64_t* bars = reinterpret_cast<uint64_t*>((reinterpret_cast<uintptr_t>(bias_part + G) + 7) & ~uintptr_t(7));  // [G]
  int* s_next = reinterpret_cast<int*>(bars + G);        // [G]
  volatile int* abort_flag = s_next + G;
  c.stage = stages + (size_t)c.gid * 3 * p.d;
  c.rounded = rounded + (size_t)c.gid * NCH * T;
  c.dots = dots + c.gid * W * 32;

  if (threadIdx.x == 0) {
    for (int i = 0; i < G; ++i) mbar_init(&bars[i], 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();

  // a kernel of this step that gave up on a bounded wait leaves stale inputs: parameters and moments stay as they are
  const bool skip = p.status != nullptr && *reinterpret_cast<const volatile int*>(p.status) != 0;
  const bool doD = p.WD != nullptr, doE = p.WE != nullptr;
  const float gmul = p.grad_mul != nullptr ? *p.grad_mul : 1.0f;
  const AdamConst h = {p.h.beta1, p.h.beta2, 1.0f - p.h.beta1, 1.0f - p.h.beta2, 1.0f / p.h.bias_correction2_sqrt,
                       p.h.lr / p.h.bias_correction1, p.h.eps};
  const bool dot_mode = p.dact_mode != 0;
  const int loadsD = p.update ? 3 : (dot_mode ? 1 : 0), loadsE = p.update ? 3 : 0;
  const uint32_t row_bytes = (uint32_t)p.d * 4u;
  float gsq = 0.0f;
  uint32_t parity = 0;  // of this group's barrier
  int red_buf = 0;

  bool outstanding = false;  // (one thread of the group) copies were issued and their arrival has not been seen
  auto issue = [&](int gid, bool is_d, int f) {  // one thread
    const int n = is_d ? loadsD : loadsE;
    if (n == 0) return;
    outstanding = true;
    uint64_t* bar = &bars[gid];
    float* dst = stages + (size_t)gid * 3 * p.d;
    mbar_arrive_expect_tx(bar, row_bytes * n);
    bulk_load(dst, (is_d ? p.WD : p.WE) + (size_t)f * p.d, row_bytes, bar);
    if (n == 3) {
      const size_t os = (size_t)(f - p.state_f0) * p.d;
      bulk_load(dst + p.d, (is_d ? p.mD : p.mE) + os, row_bytes, bar);
      bulk_load(dst + 2 * p.d, (is_d ? p.vD : p.vE) + os, row_bytes, bar);
    }
  };
  // Whether this thread has seen the copies arrive. Every caller takes a vote of all threads that share the row before anything that
  // depends on it is stored, and a group that failed draws no further rows: nothing of the side it waited for has changed then, the
  // other groups finish theirs, and the status word says that the update is incomplete.
  auto arrived = [&](int gid, uint32_t par) -> bool {
    if (p.wait_cycles > 0 && mbar_wait_bounded(&bars[gid], par, abort_flag, p.wait_cycles)) return true;
    if (c.lane == 0) report_status(const_cast<int*>(p.status), kTimeoutFullBarrier, gid);
    *abort_flag = 1;
    return false;
  };
  bool failed = false;
  auto init_grad = [&](bool is_d, int xr, float (&g)[NCH][4]) {
    const float* ex = is_d ? p.extra_gD : p.extra_gE;
#pragma unroll
    for (int i = 0; i < NCH; ++i) {
      const int col = i * W * 128 + c.tid * 4;
      float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
      if (xr >= 0 && ex != nullptr && col < p.d) e = *reinterpret_cast<const float4*>(ex + (size_t)xr * p.d + col);
      g[i][0] = e.x; g[i][1] = e.y; g[i][2] = e.z; g[i][3] = e.w;
    }
  };
  // row norm of the new decoder row (after the group barrier that follows apply_side's use of the stage)
  auto put_norm = [&](int f, float norm_sq_total) {
    if (p.norm_sq_accum != nullptr) p.norm_sq_accum[f] += norm_sq_total;  // one writer per row and launch
    else if (p.dec_norm != nullptr) p.dec_norm[f] = sqrtf(norm_sq_total);
  };
  auto put_bias = [&](int f, int xr, float bias_g) {  // one thread
    if (xr >= 0 && p.extra_gb != nullptr) bias_g += p.extra_gb[xr];
    bias_g *= gmul;
    if (p.grad_sq_sum != nullptr) gsq += bias_g * bias_g;
    if (p.update && p.bE != nullptr) {
      float b = p.bE[f], m = p.mbE[f - p.state_f0], v = p.vbE[f - p.state_f0];
      adam_update(b, m, v, bias_g, h);
      p.bE[f] = b; p.mbE[f - p.state_f0] = m; p.vbE[f - p.state_f0] = v;
    }
  };

  // several layers' rows one after the other: the group of entries and the inputs of row f
  auto group_of = [&](int f) { return p.layers_share_groups ? f % p.layer_rows : f; };
  auto inputs_of = [&](int f) { return p.layer_rows != 0 ? p.x + (size_t)(f / p.layer_rows) * p.n_rows * p.d : p.x; };

  const bool heavy_on = p.heavy != nullptr;
  // ---------------------------------------------------------------- rows with long entry lists: the whole CTA
  if (heavy_on && !skip) {
    const int n_heavy = p.heavy[0], n_long = p.layers_share_groups ? n_heavy * (p.F / p.layer_rows) : n_heavy;
    uint32_t par0 = 0;
    for (int hi = blockIdx.x; hi < n_long && !failed; hi += gridDim.x) {
      const int layer = hi / max(n_heavy, 1), group = p.heavy[1 + hi - layer * n_heavy] - p.heavy_base, f = group + layer * p.layer_rows;
      if (f < p.f_begin || f >= p.f_end) continue;
      const int e0 = p.offsets[group], e1 = p.offsets[group + 1];
      const int xr = p.extra_row != nullptr ? p.extra_row[f] : -1;
      const int rounds = (e1 - e0 + G * 32 - 1) / (G * 32), piece = (e1 - e0 + G * rounds - 1) / (G * rounds);  // (the same share to every group)
      for (int side = 0; side < 2; ++side) {
        const bool is_d = side == 0;
        if (is_d ? !doD : !doE) continue;
        if (threadIdx.x == 0) issue(0, is_d, f);
        float g[NCH][4];
        init_grad(is_d, c.gid == 0 ? xr : -1, g);
        float coef = 0.0f;
        bool seen = true;
        if (is_d) {
          if (dot_mode) {
            failed = !__syncthreads_and(arrived(0, par0));
            if (failed) break;
            round_row<W, NCH>(stages, p.d, c);
            gather_side<true, true, W, NCH>(p, c, p.dxhat, e0, e1, c.gid, G, piece, g);
          } else {
            gather_side<true, false, W, NCH>(p, c, p.dxhat, e0, e1, c.gid, G, piece, g);
          }
        } else {
          coef = gather_side<false, false, W, NCH>(p, c, inputs_of(f), e0, e1, c.gid, G, piece, g);
        }
        if (!is_d && c.wg == 0) {
          coef = warp_sum(coef);
          if (c.lane == 0) bias_part[c.gid] = coef;
        }
        if (c.gid != 0) {
#pragma unroll
          for (int i = 0; i < NCH; ++i) {
            const int col = i * W * 128 + c.tid * 4;
            if (col < p.d) *reinterpret_cast<float4*>(c.stage + col) = make_float4(g[i][0], g[i][1], g[i][2], g[i][3]);
          }
          fence_proxy_async();  // a bulk copy writes here later
        } else if ((is_d ? loadsD : loadsE) != 0 && !(is_d && dot_mode)) {
          seen = arrived(0, par0);
        }
        failed = !__syncthreads_and(seen);  // (also: the partial rows are in place)
        if (failed) break;
        if ((is_d ? loadsD : loadsE) != 0) {
          par0 ^= 1;
          if (c.gid == 0) outstanding = false;
        }
        if (c.gid == 0) {
          for (int q = 1; q < G; ++q) {
            const float* part = stages + (size_t)q * 3 * p.d;
#pragma unroll
            for (int i = 0; i < NCH; ++i) {
              const int col = i * W * 128 + c.tid * 4;
              if (col < p.d) {
                const float4 e = *reinterpret_cast<const float4*>(part + col);
                g[i][0] += e.x; g[i][1] += e.y; g[i][2] += e.z; g[i][3] += e.w;
              }
            }
          }
        }
        if (c.gid == 0) {
          if (is_d) {
            float ns = apply_side<true, W, NCH>(p, c, f, gmul, h, g, gsq);
            ns = warp_sum(ns);
            if (c.lane == 0) red[c.wg] = ns;
            group_sync<W>(0);
            if (c.tid == 0 && p.update) {
              float t = 0.0f;
              for (int w = 0; w < W; ++w) t += red[w];
              put_norm(f, t);
            }
          } else {
            apply_side<false, W, NCH>(p, c, f, gmul, h, g, gsq);
            if (c.tid == 0) {
              float b = 0.0f;
              for (int q = 0; q < G; ++q) b += bias_part[q];
              put_bias(f, xr, b);
            }
          }
        }
        __syncthreads();
      }
    }
    if (c.gid == 0) parity = par0;
  }

  // ---------------------------------------------------------------- all other rows: one group each
  int pos = 0, chunk_end = 0, turn = 0;
  auto next_row = [&]() -> int {
    if (pos + 1 < chunk_end) return ++pos;
    int b;
    if (p.sched != nullptr) {
      if constexpr (W == 1) {
        b = 0;
        if (c.lane == 0) b = atomicAdd(p.sched, p.sched_chunk);
        b = __shfl_sync(0xffffffffu, b, 0);
      } else {
        if (c.tid == 0) s_next[c.gid] = atomicAdd(p.sched, p.sched_chunk);
        group_sync<W>(c.gid);
        b = s_next[c.gid];
        group_sync<W>(c.gid);
      }
    } else {
      b = ((turn++ * G + c.gid) * (int)gridDim.x + (int)blockIdx.x) * p.sched_chunk;
    }
    pos = p.f_begin + b;
    chunk_end = min(pos + p.sched_chunk, p.f_end);
    return pos;
  };
  auto next_light = [&](int& e0, int& e1) -> int {
    int f = next_row();
    while (f < p.f_end) {
      const int group = group_of(f);
      e0 = p.offsets[group];
      e1 = p.offsets[group + 1];
      if (!heavy_on || e1 - e0 <= kHeavyRow) break;
      f = next_row();
    }
    return f;
  };

  if (!skip && !failed) {
    int e0 = 0, e1 = 0;
    int f = next_light(e0, e1);
    if (f < p.f_end && c.tid == 0) issue(c.gid, doD, f);
    while (f < p.f_end) {
      int e0n = 0, e1n = 0;
      const int fn = next_light(e0n, e1n);
      const int xr = p.extra_row != nullptr ? p.extra_row[f] : -1;
      if (doD) {
        float g[NCH][4];
        init_grad(true, xr, g);
        if (dot_mode) {
          failed = !group_all<W>(c.gid, arrived(c.gid, parity));
          if (failed) break;
          if (e1 > e0) {
            round_row<W, NCH>(c.stage, p.d, c);
            gather_side<true, true, W, NCH>(p, c, p.dxhat, e0, e1, 0, 1, 32, g);
          }
        } else {
          gather_side<true, false, W, NCH>(p, c, p.dxhat, e0, e1, 0, 1, 32, g);
        }
        if (loadsD != 0) {
          if (!dot_mode) {
            failed = !group_all<W>(c.gid, arrived(c.gid, parity));
            if (failed) break;
          }
          parity ^= 1;
          outstanding = false;
        }
        float ns = apply_side<true, W, NCH>(p, c, f, gmul, h, g, gsq);
        if (p.dec_norm != nullptr || p.norm_sq_accum != nullptr) ns = warp_sum(ns);
        float* rb = red + (red_buf * G + c.gid) * W;
        red_buf ^= 1;
        if (W > 1 && c.lane == 0) rb[c.wg] = ns;
        group_sync<W>(c.gid);  // the stage has been read
        if (c.tid == 0) {
          if (doE) issue(c.gid, false, f);
          else if (fn < p.f_end) issue(c.gid, true, fn);
          if (p.update) {
            if constexpr (W > 1) {
              ns = 0.0f;
#pragma unroll
              for (int w = 0; w < W; ++w) ns += rb[w];
            }
            put_norm(f, ns);
          }
        }
      }
      if (doE) {
        float g[NCH][4];
        init_grad(false, xr, g);
        float coef = gather_side<false, false, W, NCH>(p, c, inputs_of(f), e0, e1, 0, 1, 32, g);
        if (loadsE != 0) {
          failed = !group_all<W>(c.gid, arrived(c.gid, parity));
          if (failed) break;
          parity ^= 1;
          outstanding = false;
        }
        apply_side<false, W, NCH>(p, c, f, gmul, h, g, gsq);
        group_sync<W>(c.gid);
        if (c.tid == 0 && fn < p.f_end) issue(c.gid, doD, fn);
        if (c.wg == 0) {
          coef = warp_sum(coef);
          if (c.lane == 0) put_bias(f, xr, coef);
        }
      }
      f = fn;
      e0 = e0n;
      e1 = e1n;
    }
  }
  if (p.grad_sq_sum != nullptr) {
    gsq = warp_sum(gsq);
    if (c.lane == 0 && gsq != 0.0f) atomicAdd(p.grad_sq_sum, gsq);
  }
  // copies that nobody waited for land before the shared memory goes away
  if (failed && c.tid == 0 && outstanding) mbar_wait_bounded(&bars[c.gid], parity, nullptr);
  __syncthreads();
  if (threadIdx.x == 0 && p.sched != nullptr) {
    // the last CTA leaves the counters at zero for the next launch (every CTA has drawn its last row by then)
    __threadfence();
    if (atomicAdd(p.sched + 1, 1) == (int)gridDim.x - 1) {
      p.sched[0] = 0;
      p.sched[1] = 0;
    }
  }
}

namespace {

// A list costs one CTA 40 ns an entry in one pass with two warps a row (above 256 columns) and 26 here, and the others may have ended long before: where
// there is a longer one than this, which both kernels look at first, both sides take this kernel. 512 columns, features of popularity 1 / (5 + rank), us in
// one pass -> here: 4096 rows, 8192 tokens x 64 codes: 475 -> 340; 8192, 4096 x 64: 348 -> 255; 4096, 4096 x 32: 168 -> 115; 4096, 2048 x 64: 132 -> 105; 512,
// 2048 x 16: 69 -> 52; of equal popularity 4096, 4096 x 64: 179, 242. Batches of fewer tokens have no such list (4096, 1024 x 64: 80, 89 before
// there was the one pass) and need no second launch, which costs 1 to 2 us.
constexpr int kOnePassList = 1024;

template <int W, int NCH>
cudaError_t launch_rows(GradAdamParams p, cudaStream_t stream) {
  constexpr int T = 32 * W;
  constexpr size_t kSmemBudget = 220 * 1024;
  const size_t per_group = (size_t)p.d * 12 + (size_t)NCH * T * 8 + (size_t)W * 128 + 2 * W * 4 + 4 + 8 + 4;
  int G = (int)((kSmemBudget - 64) / per_group);
  if (G > rows_threads<NCH>() / T) G = rows_threads<NCH>() / T;
  if (W > 1 && G > 15) G = 15;  // named barriers 1..15
  if (G < 1) return cudaErrorInvalidValue;
  const int rows = p.f_end - p.f_begin;
  const int blocks = rows < 148 ? rows : 148;  // (groups without a row of their own still share the long lists)
  // rows per draw: one at the end of the range for balance, a few where rows are short and plentiful (draws are atomics on one word)
  int chunk = rows / (blocks * G * 16);
  if (p.wait_cycles < 0) p.wait_cycles = kWaitBudgetCycles;
  p.sched_chunk = chunk < 1 ? 1 : (chunk > 8 ? 8 : chunk);
  const size_t smem = (size_t)G * per_group + 64;
  auto kern = grad_adam_rows_kernel<W, NCH>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kSmemBudget + 1024));
  if (e != cudaSuccess) return e;
  launch(kern, blocks, G * T, smem, stream, p);
  return cudaGetLastError();
}

}  // namespace

// Whether this launch can take the row-streaming kernel (the CTA-per-row kernel takes the others: publication to replicas,
// dense gradient outputs, auxiliary output gradients, launches that share the SMs with another kernel).
bool grad_adam_rows_supported(const GradAdamParams& p) {
  const uintptr_t align = reinterpret_cast<uintptr_t>(p.WD) | reinterpret_cast<uintptr_t>(p.mD) | reinterpret_cast<uintptr_t>(p.vD) |
                          reinterpret_cast<uintptr_t>(p.WE) | reinterpret_cast<uintptr_t>(p.mE) | reinterpret_cast<uintptr_t>(p.vE);
  return p.d % 4 == 0 && p.d <= 8192 && p.n_pub == 0 && p.gD_out == nullptr && p.gE_out == nullptr && p.ctas_per_sm == 0 &&
         p.dxhat_aux == nullptr && align % 16 == 0;
}

int grad_adam_rows_launch(GradAdamParams p, cudaStream_t stream) {
  if (!grad_adam_rows_supported(p) || (p.dact_mode != 0 && (p.WD == nullptr || p.dact_out == nullptr))) return (int)cudaErrorInvalidValue;
  if (p.f_end <= p.f_begin) return 0;
  const int d = p.d;
  cudaError_t e;
  if (grad_adam_both_supported(p)) {
    const bool either = d > 256 && p.heavy != nullptr && p.n_rows > kOnePassList;
    p.longest = either ? kOnePassList : 0;
    const int err = grad_adam_both_launch(p, stream);
    if (err != 0 || !either) return err;
    p.longest = -kOnePassList;
  }
  if (d <= 1024) {
    const int nch = (d + 127) / 128;
    e = nch <= 1 ? launch_rows<1, 1>(p, stream) : nch <= 2 ? launch_rows<1, 2>(p, stream) : nch <= 4 ? launch_rows<1, 4>(p, stream)
        : nch <= 6 ? launch_rows<1, 6>(p, stream) : launch_rows<1, 8>(p, stream);
  } else if (d <= 2048) {
    e = d <= 1536 ? launch_rows<2, 6>(p, stream) : launch_rows<2, 8>(p, stream);
  } else if (d <= 4096) {
    e = d <= 3072 ? launch_rows<4, 6>(p, stream) : launch_rows<4, 8>(p, stream);
  } else {
    e = d <= 6144 ? launch_rows<8, 6>(p, stream) : launch_rows<8, 8>(p, stream);
  }
  return (int)e;
}

}  // namespace lmsae
