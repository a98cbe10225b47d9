// Warp-level gather of weighted bf16 rows: the inner loop of the sparse decoders.
#pragma once
#include "common.cuh"

namespace lmsae {

__device__ __forceinline__ void bf16x8_to_float(const uint4& u, float (&f)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    f[2 * i] = __uint_as_float(w[i] << 16);
    f[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}

// (d0, d1) += (a0, a1) * (b0, b1) in one instruction
__device__ __forceinline__ void fma2(float& d0, float& d1, float a0, float a1, float b0, float b1) {
  asm("{\n\t"
      ".reg .b64 ra, rb, rd;\n\t"
      "mov.b64 ra, {%2, %3};\n\t"
      "mov.b64 rb, {%4, %5};\n\t"
      "mov.b64 rd, {%0, %1};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rd;\n\t"
      "mov.b64 {%0, %1}, rd;\n\t"
      "}"
      : "+f"(d0), "+f"(d1)
      : "f"(a0), "f"(a1), "f"(b0), "f"(b1));
}

// acc[u][:] = sum_j val[j] * W[idx[j], 8 v[u] .. 8 v[u] + 8) over the entries of one list (idx < 0: empty slot; idx >= limit:
// not for this caller), lanes of the warp owning the 16-byte chunks v[u] of every row. Lanes fetch 32 entries at a time
// (the next 32 while the rows of these are on their way) and hand them round by shuffles; the rows of up to eight
// entries (four for VPT = 2) are requested before the first is used. An entry whose coefficient is zero counts like any other: a row that
// is not finite shows in the sum (passing over them instead saved nothing: a crosscoder step of 8 heads takes 16.29 ms either way).
template <int VPT>
__device__ __forceinline__ void gather_rows_warp(const int* __restrict__ idx, const float* __restrict__ val, int k,
                                                 const __nv_bfloat16* __restrict__ W, int d, long long n_rows, long long limit,
                                                 const int (&v)[VPT], const bool (&in)[VPT], float (&acc)[VPT][8]) {
  constexpr int U = 8 / VPT;
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int u = 0; u < VPT; ++u)
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[u][i] = 0.0f;
  int f_next = -1;
  float a_next = 0.0f;
  if (lane < k) { f_next = __ldg(idx + lane); a_next = __ldg(val + lane); }
  for (int base = 0; base < k; base += 32) {
    const int f_l = f_next;
    const float a_l = a_next;
    f_next = -1;
    if (base + 32 + lane < k) { f_next = __ldg(idx + base + 32 + lane); a_next = __ldg(val + base + 32 + lane); }
    unsigned mask = __ballot_sync(0xffffffffu, f_l >= 0 && f_l < limit);
    while (mask != 0u) {  // (the mask is the same in every lane)
      uint4 w[U][VPT];
      float a[U];
#pragma unroll
      for (int e = 0; e < U; ++e) {
        a[e] = 0.0f;
        if (mask != 0u) {
          const int j = __ffs(mask) - 1;
          mask &= mask - 1u;
          const int f = __shfl_sync(0xffffffffu, f_l, j);
          a[e] = __shfl_sync(0xffffffffu, a_l, j);
          const uint4* row = reinterpret_cast<const uint4*>(W + (size_t)LMSAE_IDX(f, n_rows) * d);
#pragma unroll
          for (int u = 0; u < VPT; ++u) w[e][u] = in[u] ? __ldg(row + v[u]) : make_uint4(0u, 0u, 0u, 0u);
        } else {
#pragma unroll
          for (int u = 0; u < VPT; ++u) w[e][u] = make_uint4(0u, 0u, 0u, 0u);
        }
      }
#pragma unroll
      for (int e = 0; e < U; ++e) {
#pragma unroll
        for (int u = 0; u < VPT; ++u) {
          float x[8];
          bf16x8_to_float(w[e][u], x);
#pragma unroll
          for (int i = 0; i < 8; i += 2) fma2(acc[u][i], acc[u][i + 1], x[i], x[i + 1], a[e], a[e]);
        }
      }
    }
  }
}

}  // namespace lmsae
