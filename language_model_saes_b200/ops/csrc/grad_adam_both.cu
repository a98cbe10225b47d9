// Sparse gradient rows + Adam for both sides of a dictionary with short rows, in one pass over a feature's entries (sm_100a).
//
// Same result as grad_adam.cu, which says what is computed. There the decoder side of a row is gathered, applied and stored before its
// encoder side begins, since the code gradients that the encoder side multiplies come from the decoder side's dot products. A row's
// time is then twice the chain entry -> code -> gathered rows -> Adam, and with short rows such chains are what the kernel takes: 4096 rows
// of 512 with up to 21 (35) entries took 45 (50) us of which the bytes need 17.
// Here a token's row of d x_hat and its row of x are requested together. The dot product of the first with the decoder row is the
// coefficient of the second, so that one round trip serves both sides; the rows' six streams (p, m, v of both sides) are fetched at once.
//   group of W warps   one feature row; a thread owns four columns (NCH of them, 128 W apart), W = ceil(d / (128 NCH))
//   Q entries          at a time: 2 Q NCH 8-byte loads in flight per thread. The Q dot products are reduced together (nine shuffles for
//                      eight sums instead of forty), across the group's warps through shared memory behind one barrier
//   ahead of the row   the entries and codes of the next row, the range of the one after it and its draw from the row counter are requested
//                      while this one's gathers are on their way
//   long lists         as in grad_adam.cu, the same share to every group, a piece's entries and codes requested while the ones before it are gathered (in pieces
//                      of eight, each behind the one before it: 4096 rows of 512, 4096 x 64 codes 187 us, 175 here; skewed popularity, 4096 x 32: 186, 168)
// Bound by instructions and their latency (0.42 issued per cycle and scheduler, a thousand per row and warp with an entry or two), not by memory.
// grad_adam.cu -> this, us; up to 128 columns NCH 1, Q 8, above NCH 2, Q 4 (in brackets the other of the two):
//   256 x 64, 512 tokens x 8 codes        24.5 -> 15.6 (18.5)     512 x 128, 2048 x 16     41.0 -> 28.6 (36.9)
//   1024 x 64, 700 x 11                   21.4 -> 13.5 (15.4)     2048 x 256, 1024 x 32    35.8 -> 21.4 (22.6)
//   8592 x 104, 702 x 11                  30.7 -> 24.6 (24.6)     4096 x 512, 1024 x 32    45.1 -> 36.9 (43.9)
//   16384 x 256, 4096 x 32                65.6 -> 58.4 (72.6)
// Wider rows stay where they are: they keep more loads in flight per instruction there, and their streams bind (24576 x 768, 4096 x 50: 194 us,
// here 227; 7376 x 1024, 2016 x 47: 104, 114). A second set of stages for the next row's streams changed nothing (36.9 -> 38.1).
#include "adam.cuh"
#include "gather.cuh"
#include "kernels.h"

namespace lmsae {

LMSAE_DEFINE_BOUNDS_FETCH(bounds_fetch_grad_adam_both)

namespace {

constexpr int GB_THREADS = 512;  // (128 registers: nothing is spilled)

struct BothCtx {
  int gid, wg, lane, tid, W;  // group, warp within it, lane, thread within it, warps of a group
  float* stage;               // [6][d]: parameter and moments of the decoder row, then of the encoder row
  float* dots;                // [2][W][8] partial dot products
};

__device__ __forceinline__ void group_sync(const BothCtx& c) {
  if (c.W == 1) __syncwarp();
  else asm volatile("bar.sync %0, %1;" ::"r"(c.gid + 1), "r"(c.W * 32) : "memory");
}
// Whether all threads of the group say so (a barrier of the group).
__device__ __forceinline__ bool group_all(const BothCtx& c, bool ok) {
  if (c.W == 1) return __all_sync(0xffffffffu, ok);
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
      : "r"(c.gid + 1), "r"(c.W * 32), "r"((uint32_t)ok)
      : "memory");
  return r != 0;
}

// Sums of v[0..Q) over the warp; lane l ends with the one of q = l / (32 / Q).
template <int Q>
__device__ __forceinline__ float warp_sums(float (&v)[Q], int lane) {
#pragma unroll
  for (int n = Q / 2, o = 16; n >= 1; n /= 2, o /= 2) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float give = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
#pragma unroll
  for (int o = 16 / Q; o >= 1; o /= 2) v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
  return v[0];
}

// A lane's entry of the list: its position, its token and its code
struct Entry {
  int at, row;
  float a;
};
__device__ __forceinline__ int entry_at(const GradAdamParams& p, int e, int n, int lane) {
  return lane < n ? (int)LMSAE_IDX(p.entries[e + lane], p.n_codes) : 0;
}
__device__ __forceinline__ Entry entry_of(const GradAdamParams& p, int at, int n, int lane) {
  Entry m = {at, (int)LMSAE_IDX(at / p.k, p.n_rows), 0.0f};
  if (lane < n) m.a = p.act[at];
  return m;
}

// Adds the entries [e, e + n), n <= 32, of one feature to both of its gradient rows, and their code gradients to `coef`.
template <int NCH, int Q>
__device__ __forceinline__ void gather_both(const GradAdamParams& p, const BothCtx& c, const Entry& m, int n, const uint2 (&w)[NCH], float (&gD)[NCH][4],
                                            float (&gE)[NCH][4], float& coef, int& buf) {
  unsigned mask = __ballot_sync(0xffffffffu, m.a != 0.0f);  // (the same in every warp of the group)
  float dact = 0.0f;
  while (mask != 0u) {
    int j[Q];
    float a[Q];
    uint2 ud[Q][NCH], ux[Q][NCH];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      j[q] = -1;
      a[q] = 0.0f;
#pragma unroll
      for (int i = 0; i < NCH; ++i) ud[q][i] = ux[q][i] = make_uint2(0u, 0u);
      if (mask != 0u) {
        j[q] = __ffs(mask) - 1;
        mask &= mask - 1u;
        a[q] = __shfl_sync(0xffffffffu, m.a, j[q]);
        const size_t o = (size_t)__shfl_sync(0xffffffffu, m.row, j[q]) * p.d + c.tid * 4;
#pragma unroll
        for (int i = 0; i < NCH; ++i)
          if (i * c.W * 128 + c.tid * 4 < p.d) {
            ud[q][i] = __ldg(reinterpret_cast<const uint2*>(p.dxhat + o + i * c.W * 128));
            ux[q][i] = __ldg(reinterpret_cast<const uint2*>(p.x + o + i * c.W * 128));
          }
      }
    }
    float s[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      float d0 = 0.0f, d1 = 0.0f;
#pragma unroll
      for (int i = 0; i < NCH; ++i) {
        const float x0 = __uint_as_float(ud[q][i].x << 16), x1 = __uint_as_float(ud[q][i].x & 0xffff0000u);
        const float x2 = __uint_as_float(ud[q][i].y << 16), x3 = __uint_as_float(ud[q][i].y & 0xffff0000u);
        fma2(gD[i][0], gD[i][1], x0, x1, a[q], a[q]);
        fma2(gD[i][2], gD[i][3], x2, x3, a[q], a[q]);
        fma2(d0, d1, x0, x1, __uint_as_float(w[i].x << 16), __uint_as_float(w[i].x & 0xffff0000u));
        fma2(d0, d1, x2, x3, __uint_as_float(w[i].y << 16), __uint_as_float(w[i].y & 0xffff0000u));
      }
      s[q] = d0 + d1;
    }
    const float mine = warp_sums<Q>(s, c.lane);
    float* dots = c.dots + buf * c.W * 8;  // (the other one may still be read)
    buf ^= 1;
    if (c.lane % (32 / Q) == 0) dots[c.wg * 8 + c.lane / (32 / Q)] = mine;
    group_sync(c);
    float dot[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) dot[q] = 0.0f;
    for (int g = 0; g < c.W; ++g) {
#pragma unroll
      for (int q = 0; q < Q; q += 4) {
        const float4 t = *reinterpret_cast<const float4*>(dots + g * 8 + q);
        dot[q] += t.x; dot[q + 1] += t.y; dot[q + 2] += t.z; dot[q + 3] += t.w;
      }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      if (c.lane == j[q]) dact = dot[q];
      if (j[q] < 0 || dot[q] == 0.0f) continue;  // (the same in every thread of the group; a code gradient of 0 takes nothing of its row)
      coef += dot[q];
#pragma unroll
      for (int i = 0; i < NCH; ++i) {
        fma2(gE[i][0], gE[i][1], __uint_as_float(ux[q][i].x << 16), __uint_as_float(ux[q][i].x & 0xffff0000u), dot[q], dot[q]);
        fma2(gE[i][2], gE[i][3], __uint_as_float(ux[q][i].y << 16), __uint_as_float(ux[q][i].y & 0xffff0000u), dot[q], dot[q]);
      }
    }
  }
  if (c.wg == 0 && c.lane < n) p.dact_out[m.at] = dact;  // (0 where the code is)
}

}  // namespace

template <int NCH, int Q>
__global__ void __launch_bounds__(GB_THREADS, 1)
grad_adam_both_kernel(const GradAdamParams p, const int W) {
  pdl_wait();
  if (p.longest > 0 && any_longer_list(p, p.longest)) return;  // (the launch of the other kernel does it)
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const int T = 32 * W, G = (int)blockDim.x / T, d = p.d;
  BothCtx c;
  c.W = W;
  c.gid = (int)threadIdx.x / T;
  c.tid = (int)threadIdx.x % T;
  c.wg = c.tid >> 5;
  c.lane = (int)threadIdx.x & 31;
  float* stages = reinterpret_cast<float*>(smem_raw);
  float* all_dots = stages + (size_t)G * 6 * d;        // [G][2][W][8]
  float* red = all_dots + (size_t)G * 2 * W * 8;       // [2][G][W] norms, then [G] bias sums
  float* bias_part = red + 2 * G * W;
  uint64_t* bars = reinterpret_cast<uint64_t*>((reinterpret_cast<uintptr_t>(bias_part + G) + 7) & ~uintptr_t(7));  // [G]
  int* s_next = reinterpret_cast<int*>(bars + G);      // [2][G]
  volatile int* abort_flag = s_next + 2 * G;
  c.stage = stages + (size_t)c.gid * 6 * d;
  c.dots = all_dots + (size_t)c.gid * 2 * W * 8;

  if (threadIdx.x == 0) {
    for (int i = 0; i < G; ++i) mbar_init(&bars[i], 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();

  // a kernel of this step that gave up on a bounded wait leaves stale inputs: parameters and moments stay as they are
  const bool skip = p.status != nullptr && *reinterpret_cast<const volatile int*>(p.status) != 0;
  const float gmul = p.grad_mul != nullptr ? *p.grad_mul : 1.0f;
  const AdamConst h = {p.h.beta1, p.h.beta2, 1.0f - p.h.beta1, 1.0f - p.h.beta2, 1.0f / p.h.bias_correction2_sqrt,
                       p.h.lr / p.h.bias_correction1, p.h.eps};
  const uint32_t row_bytes = (uint32_t)d * 4u;
  uint32_t parity = 0;  // of this group's barrier
  int dot_buf = 0, red_buf = 0;
  bool failed = false, outstanding = false;  // (outstanding: one thread of the group issued copies whose arrival has not been seen)

  auto issue = [&](int gid, int f) {  // one thread
    outstanding = true;
    uint64_t* bar = &bars[gid];
    float* dst = stages + (size_t)gid * 6 * d;
    const size_t o = (size_t)f * d, os = (size_t)(f - p.state_f0) * d;
    mbar_arrive_expect_tx(bar, row_bytes * 6);
    bulk_load(dst, p.WD + o, row_bytes, bar);
    bulk_load(dst + d, p.mD + os, row_bytes, bar);
    bulk_load(dst + 2 * d, p.vD + os, row_bytes, bar);
    bulk_load(dst + 3 * d, p.WE + o, row_bytes, bar);
    bulk_load(dst + 4 * d, p.mE + os, row_bytes, bar);
    bulk_load(dst + 5 * d, p.vE + os, row_bytes, bar);
  };
  // Whether this thread has seen the copies arrive. Every caller takes a vote of all threads that share the row before anything that
  // depends on it is stored, and a group that failed takes no further rows: nothing of that row has changed then, the other groups
  // finish theirs, and the status word says that the update is incomplete.
  auto arrived = [&](int gid, uint32_t par) -> bool {
    if (p.wait_cycles > 0 && mbar_wait_bounded(&bars[gid], par, abort_flag, p.wait_cycles)) return true;
    if (c.lane == 0) report_status(const_cast<int*>(p.status), kTimeoutFullBarrier, gid);
    *abort_flag = 1;
    return false;
  };
  auto init_grad = [&](const float* extra, int xr, float (&g)[NCH][4]) {
#pragma unroll
    for (int i = 0; i < NCH; ++i) {
      const int col = i * T * 4 + c.tid * 4;
      float4 e = make_float4(0.f, 0.f, 0.f, 0.f);
      if (xr >= 0 && extra != nullptr && col < d) e = *reinterpret_cast<const float4*>(extra + (size_t)xr * d + col);
      g[i][0] = e.x; g[i][1] = e.y; g[i][2] = e.z; g[i][3] = e.w;
    }
  };
  // the bf16-rounded decoder row that the forward pass used (what the shadow holds)
  auto rounded_row = [&](const float* row, uint2 (&w)[NCH]) {
#pragma unroll
    for (int i = 0; i < NCH; ++i) {
      const int col = i * T * 4 + c.tid * 4;
      w[i] = make_uint2(0u, 0u);  // (columns past the end multiply zeros: they must not hold a NaN)
      if (col < d) {
        const float4 v = *reinterpret_cast<const float4*>(row + col);
        w[i] = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
      }
    }
  };
  // Adam on one side of row f from its staged streams; returns this thread's share of the new row's squared norm
  auto apply = [&](bool is_d, int f, const float* st, float (&g)[NCH][4]) {
    float* Wp = is_d ? p.WD : p.WE;
    float* Mp = is_d ? p.mD : p.mE;
    float* Vp = is_d ? p.vD : p.vE;
    __nv_bfloat16* Sp = is_d ? p.WD_bf16 : p.WE_bf16;
    const size_t o = (size_t)f * d, os = (size_t)(f - p.state_f0) * d;
    const float self_scale = (is_d && p.wd_self_scale != nullptr) ? p.wd_self_scale[f] * gmul : 0.0f;
    float norm_sq = 0.0f;
#pragma unroll
    for (int i = 0; i < NCH; ++i) {
      const int col = i * T * 4 + c.tid * 4;
      if (col >= d) continue;
      float4 w = *reinterpret_cast<const float4*>(st + col);
      float4 m = *reinterpret_cast<const float4*>(st + d + col);
      float4 v = *reinterpret_cast<const float4*>(st + 2 * d + col);
#pragma unroll
      for (int q = 0; q < 4; ++q) g[i][q] *= gmul;
      if (is_d) {
        g[i][0] = fmaf(self_scale, w.x, g[i][0]); g[i][1] = fmaf(self_scale, w.y, g[i][1]);
        g[i][2] = fmaf(self_scale, w.z, g[i][2]); g[i][3] = fmaf(self_scale, w.w, g[i][3]);
      }
      adam_update(w.x, m.x, v.x, g[i][0], h); adam_update(w.y, m.y, v.y, g[i][1], h);
      adam_update(w.z, m.z, v.z, g[i][2], h); adam_update(w.w, m.w, v.w, g[i][3], h);
      __stcs(reinterpret_cast<float4*>(Wp + o + col), w);
      __stcs(reinterpret_cast<float4*>(Mp + os + col), m);
      __stcs(reinterpret_cast<float4*>(Vp + os + col), v);
      norm_sq += w.x * w.x + w.y * w.y + w.z * w.z + w.w * w.w;
      *reinterpret_cast<uint2*>(Sp + o + col) = make_uint2(pack_bf16x2(w.x, w.y), pack_bf16x2(w.z, w.w));
    }
    return norm_sq;
  };
  auto put_norm = [&](int f, const float* parts) {  // one thread
    if (p.dec_norm == nullptr) return;
    float t = 0.0f;
    for (int w = 0; w < W; ++w) t += parts[w];
    p.dec_norm[f] = sqrtf(t);
  };
  auto put_bias = [&](int f, int xr, float g, float b, float m, float v) {  // one thread
    if (xr >= 0 && p.extra_gb != nullptr) g += p.extra_gb[xr];
    adam_update(b, m, v, g * gmul, h);
    p.bE[f] = b; p.mbE[f - p.state_f0] = m; p.vbE[f - p.state_f0] = v;
  };

  const bool heavy_on = p.heavy != nullptr;
  // ---------------------------------------------------------------- rows with long entry lists: the whole CTA
  if (heavy_on && !skip) {
    const int n_heavy = p.heavy[0];
    for (int hi = blockIdx.x; hi < n_heavy; hi += gridDim.x) {
      const int f = p.heavy[1 + hi] - p.heavy_base;
      if (f < p.f_begin || f >= p.f_end) continue;
      const int e0 = p.offsets[f], e1 = p.offsets[f + 1];
      const int xr = p.extra_row != nullptr ? p.extra_row[f] : -1;
      if (threadIdx.x == 0) issue(0, f);
      // the same share to every group, in pieces of at most 32 entries; a piece's entries are requested two pieces ahead of it, its codes one
      const int n = e1 - e0, rounds = (n + G * 32 - 1) / (G * 32), piece = (n + G * rounds - 1) / (G * rounds), step = G * piece;
      auto left = [&](int i) { return max(0, min(piece, n - i)); };
      int i0 = c.gid * piece;
      Entry m = entry_of(p, entry_at(p, e0 + i0, left(i0), c.lane), left(i0), c.lane);
      int at_n = entry_at(p, e0 + i0 + step, left(i0 + step), c.lane);
      float gD[NCH][4], gE[NCH][4], coef = 0.0f;
      uint2 w[NCH];
      init_grad(p.extra_gD, c.gid == 0 ? xr : -1, gD);
      init_grad(p.extra_gE, c.gid == 0 ? xr : -1, gE);
      // (bars[0] is group 0's, whose parity the others follow in `parity` until the lists are done)
      failed = !__syncthreads_and(arrived(0, parity));
      if (failed) break;
      parity ^= 1;
      outstanding = false;
      rounded_row(stages, w);
      for (; i0 < n; i0 += step) {
        const Entry next = entry_of(p, at_n, left(i0 + step), c.lane);
        at_n = entry_at(p, e0 + i0 + 2 * step, left(i0 + 2 * step), c.lane);
        gather_both<NCH, Q>(p, c, m, left(i0), w, gD, gE, coef, dot_buf);
        m = next;
      }
      if (c.tid == 0) bias_part[c.gid] = coef;
      if (c.gid != 0) {
#pragma unroll
        for (int i = 0; i < NCH; ++i) {
          const int col = i * T * 4 + c.tid * 4;
          if (col < d) {
            *reinterpret_cast<float4*>(c.stage + col) = make_float4(gD[i][0], gD[i][1], gD[i][2], gD[i][3]);
            *reinterpret_cast<float4*>(c.stage + d + col) = make_float4(gE[i][0], gE[i][1], gE[i][2], gE[i][3]);
          }
        }
        fence_proxy_async();  // a bulk copy writes here later
      }
      __syncthreads();
      if (c.gid == 0) {
        for (int q = 1; q < G; ++q) {
          const float* part = stages + (size_t)q * 6 * d;
#pragma unroll
          for (int i = 0; i < NCH; ++i) {
            const int col = i * T * 4 + c.tid * 4;
            if (col < d) {
              const float4 a = *reinterpret_cast<const float4*>(part + col), b = *reinterpret_cast<const float4*>(part + d + col);
              gD[i][0] += a.x; gD[i][1] += a.y; gD[i][2] += a.z; gD[i][3] += a.w;
              gE[i][0] += b.x; gE[i][1] += b.y; gE[i][2] += b.z; gE[i][3] += b.w;
            }
          }
        }
        const float ns = warp_sum(apply(true, f, stages, gD));
        apply(false, f, stages + 3 * d, gE);
        if (c.lane == 0) red[c.wg] = ns;
        group_sync(c);
        if (c.tid == 0) {
          put_norm(f, red);
          if (p.bE != nullptr) {
            float b = 0.0f;
            for (int q = 0; q < G; ++q) b += bias_part[q];
            put_bias(f, xr, b, p.bE[f], p.mbE[f - p.state_f0], p.vbE[f - p.state_f0]);
          }
        }
      }
      __syncthreads();
    }
    if (c.gid != 0) parity = 0;
  }

  // ---------------------------------------------------------------- all other rows: one group each
  // Pieces of sched_chunk rows: a group's first two are dealt out, the others drawn, so that the wait for a draw is never in the way.
  const int n_groups = G * (int)gridDim.x;
  int pos = 0, piece_end = 0, turn = 0;
  auto next_is_drawn = [&] { return pos + 1 >= piece_end && turn >= 2 && p.sched != nullptr && pos < p.f_end; };
  auto next_row = [&](int drawn) {
    if (pos + 1 < piece_end) return ++pos;
    if (turn >= 2 && pos >= p.f_end) return pos;
    const int b = turn < 2 || p.sched == nullptr ? (turn * n_groups + c.gid * (int)gridDim.x + (int)blockIdx.x) * p.sched_chunk
                                                 : 2 * n_groups * p.sched_chunk + drawn;
    ++turn;
    pos = p.f_begin + min(b, p.f_end - p.f_begin);
    piece_end = min(pos + p.sched_chunk, p.f_end);
    return pos;
  };
  auto range_of = [&](int f, int& e0, int& e1) {
    e0 = e1 = 0;
    if (f < p.f_end) { e0 = p.offsets[f]; e1 = p.offsets[f + 1]; }
  };
  auto is_light = [&](int f, int n) { return f < p.f_end && (!heavy_on || n <= kHeavyRow); };

  if (!skip && !failed) {
    int e0, e1, e0n, e1n;
    int f = next_row(0);
    range_of(f, e0, e1);
    // (with a piece of more than one row the second row is in the same piece, and the second piece still dealt out)
    int fn = f < p.f_end ? next_row(0) : f;
    range_of(fn, e0n, e1n);
    if (is_light(f, e1 - e0) && c.tid == 0) issue(c.gid, f);
    int n = is_light(f, e1 - e0) ? min(32, e1 - e0) : 0;
    Entry m = entry_of(p, entry_at(p, e0, n, c.lane), n, c.lane);
    while (f < p.f_end) {
      const int nn = is_light(fn, e1n - e0n) ? min(32, e1n - e0n) : 0;
      const int at_n = entry_at(p, e0n, nn, c.lane);
      const bool draws = next_is_drawn();
      int drawn = 0;
      if (draws && c.tid == 0) drawn = atomicAdd(p.sched, p.sched_chunk);
      float* rb = red + (red_buf * G + c.gid) * W;  // (two of each in turn: the other may still be read)
      int* drawn_s = s_next + red_buf * G + c.gid;
      red_buf ^= 1;
      const bool light = is_light(f, e1 - e0);
      float coef = 0.0f, ns = 0.0f, b = 0.0f, bm = 0.0f, bv = 0.0f;
      int xr = -1;
      if (light) {
        xr = p.extra_row != nullptr ? p.extra_row[f] : -1;
        if (c.tid == 0 && p.bE != nullptr) { b = p.bE[f]; bm = p.mbE[f - p.state_f0]; bv = p.vbE[f - p.state_f0]; }
        float gD[NCH][4], gE[NCH][4];
        uint2 w[NCH];
        init_grad(p.extra_gD, xr, gD);
        init_grad(p.extra_gE, xr, gE);
        failed = !group_all(c, arrived(c.gid, parity));
        if (failed) break;
        parity ^= 1;
        outstanding = false;
        rounded_row(c.stage, w);
        gather_both<NCH, Q>(p, c, m, n, w, gD, gE, coef, dot_buf);
        for (int e = e0 + 32; e < e1; e += 32) {
          const int more = min(32, e1 - e);
          gather_both<NCH, Q>(p, c, entry_of(p, entry_at(p, e, more, c.lane), more, c.lane), more, w, gD, gE, coef, dot_buf);
        }
        ns = apply(true, f, c.stage, gD);
        apply(false, f, c.stage + 3 * d, gE);
        if (p.dec_norm != nullptr) ns = warp_sum(ns);
        if (c.lane == 0) rb[c.wg] = ns;
      }
      m = entry_of(p, at_n, nn, c.lane);
      if (draws && c.tid == 0) *drawn_s = drawn;
      group_sync(c);  // the stage has been read
      if (c.tid == 0) {
        if (is_light(fn, e1n - e0n)) issue(c.gid, fn);
        if (light) {
          put_norm(f, rb);
          if (p.bE != nullptr) put_bias(f, xr, coef, b, bm, bv);
        }
      }
      const int f2 = next_row(draws ? *drawn_s : 0);
      f = fn; e0 = e0n; e1 = e1n; n = nn;
      fn = f2;
      range_of(fn, e0n, e1n);
    }
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

template <int NCH, int Q>
static cudaError_t launch_both(GradAdamParams p, cudaStream_t stream) {
  constexpr size_t kSmemBudget = 220 * 1024;
  const int W = (p.d + 128 * NCH - 1) / (128 * NCH), T = 32 * W;
  const size_t per_group = (size_t)p.d * 24 + (size_t)W * 64 + 2 * W * 4 + 4 + 8 + 8;
  int G = (int)((kSmemBudget - 64) / per_group);
  if (G > GB_THREADS / T) G = GB_THREADS / T;
  if (W > 1 && G > 15) G = 15;  // named barriers 1..15
  if (G < 1) return cudaErrorInvalidValue;
  const int rows = p.f_end - p.f_begin;
  const int blocks = rows < 148 ? rows : 148;  // (groups without a row of their own still share the long lists)
  // rows per draw: one at the end of the range for balance, a few where rows are short and plentiful (draws are atomics on one word)
  const int chunk = rows / (blocks * G * 16);
  p.sched_chunk = chunk < 1 ? 1 : (chunk > 8 ? 8 : chunk);
  if (p.wait_cycles < 0) p.wait_cycles = kWaitBudgetCycles;
  const cudaError_t e = cudaFuncSetAttribute(grad_adam_both_kernel<NCH, Q>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kSmemBudget + 1024));
  if (e != cudaSuccess) return e;
  launch(grad_adam_both_kernel<NCH, Q>, blocks, G * T, (size_t)G * per_group + 64, stream, p, W);
  return cudaGetLastError();
}

// Whether grad_adam_rows_launch hands this launch on: short rows, both sides and their code gradients at once, parameters updated, nothing
// else asked for.
bool grad_adam_both_supported(const GradAdamParams& p) {
  return p.WD != nullptr && p.WE != nullptr && p.dact_mode == 1 && p.update && p.grad_sq_sum == nullptr && p.norm_sq_accum == nullptr && p.layer_rows == 0 &&
         p.d <= 512;
}

int grad_adam_both_launch(const GradAdamParams& p, cudaStream_t stream) {
  return (int)(p.d <= 128 ? launch_both<1, 8>(p, stream) : launch_both<2, 4>(p, stream));
}

}  // namespace lmsae
