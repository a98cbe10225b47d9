// fp32 products of listed rows on the fp32 pipes (sm_100a): what the sparse and the estimating kernels of inference leave over. The
// list is made on the device and is empty as a rule: the launch then ends at once, and the host never waits for its length.
//
//   C[r, n] = sum_k A[r, k] * B[n, k]  or  sum_k A[r, k] * B[k, n]   for every r of the list
//
// 128 x 128 tiles, eight rows x eight columns a thread, sums in ascending order of k, one rounding per term (fma). Persistent CTAs,
// two to an SM. With `part`, k is cut into as many slices as fill the GPU evenly; the last CTA of a tile adds the slices up in order.
#include "gather.cuh"
#include "kernels.h"

namespace lmsae {

namespace {

constexpr int RP_M = 128, RP_N = 128, RP_K = 16, RP_THREADS = 256, RP_LD = 132;
constexpr int RP_SLOTS = 148 * 2;

template <bool B_BY_K>  // B is [K, N] (else [N, K])
__global__ void __launch_bounds__(RP_THREADS, 2)
rows_product_kernel(const RowsProductParams p) {
  pdl_wait();
  __shared__ __align__(16) float s_a[2][RP_K][RP_LD];
  __shared__ __align__(16) float s_b[2][RP_K][RP_LD];
  __shared__ int s_last, s_every;
  if (threadIdx.x == 0) s_every = p.every != nullptr && *p.every != 0;
  __syncthreads();
  const int n_rows = s_every ? p.max_rows : p.rows[0];
  if (n_rows == 0) return;
  // (the choice stays in shared memory: a register more for the whole loop spills 190 bytes, and 4096 rows of 24576 x 768 take 5.6 ms instead of 4.7)
  auto row_at = [&](int r) { return s_every ? r : p.rows[1 + r]; };
  const int mt = (n_rows + RP_M - 1) / RP_M, nt = (p.N + RP_N - 1) / RP_N, tiles = mt * nt;
  const int k_blocks = (p.K + RP_K - 1) / RP_K;
  int slices = 1;
  if (p.part != nullptr && tiles < 4 * RP_SLOTS) {  // the number whose last wave is the fullest
    float best = 1e30f;
    for (int s = 1; s <= 16; ++s) {
      if ((long long)s * tiles * RP_M * RP_N > p.part_floats || tiles > p.part_tiles || s * 8 > k_blocks) break;
      const float cost = (float)((tiles * s + RP_SLOTS - 1) / RP_SLOTS) / (float)s + 0.004f * (float)(s - 1);
      if (cost < best) { best = cost; slices = s; }
    }
  }
  const int tid = threadIdx.x;
  const int lr = tid & 127, lk = (tid >> 7) * 8;      // row of A (of B) and first k that this thread fetches
  const int bk = tid >> 5, bn = (tid & 31) * 4;       // B by k: k (and k + 8) and columns
  const int ty = (tid >> 4) * 4, tx = (tid & 15) * 4;  // rows ty.., 64 + ty.., columns tx.., 64 + tx..
  for (int item = blockIdx.x; item < tiles * slices; item += gridDim.x) {
    const int slice = item / tiles, tile = item - slice * tiles;
    const int m0 = (tile % mt) * RP_M, n0 = (tile / mt) * RP_N;
    const int kb0 = (int)((long long)k_blocks * slice / slices), kb1 = (int)((long long)k_blocks * (slice + 1) / slices);
    const float* a_row = m0 + lr < n_rows ? p.A + (size_t)row_at(m0 + lr) * p.K : nullptr;
    const float* b_row = !B_BY_K && n0 + lr < p.N ? p.B + (size_t)(n0 + lr) * p.K : nullptr;
    float4 ra[2], rb[2];
    auto fetch = [&](int kb) {
      const int k0 = kb * RP_K;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int k = k0 + lk + i * 4;  // (K % 4 == 0)
        ra[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        rb[i] = ra[i];
        if (a_row != nullptr && k < p.K) ra[i] = __ldg(reinterpret_cast<const float4*>(a_row + k));
        if constexpr (B_BY_K) {
          const int kk = k0 + bk + i * 8;  // (N % 4 == 0)
          if (kk < p.K && n0 + bn < p.N) rb[i] = __ldg(reinterpret_cast<const float4*>(p.B + (size_t)kk * p.N + n0 + bn));
        } else if (b_row != nullptr && k < p.K) {
          rb[i] = __ldg(reinterpret_cast<const float4*>(b_row + k));
        }
      }
    };
    auto put = [&](int buf) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        float(*a)[RP_LD] = s_a[buf];
        const int k = lk + i * 4;
        a[k][lr] = ra[i].x; a[k + 1][lr] = ra[i].y; a[k + 2][lr] = ra[i].z; a[k + 3][lr] = ra[i].w;
        float(*b)[RP_LD] = s_b[buf];
        if constexpr (B_BY_K) {
          *reinterpret_cast<float4*>(&b[bk + i * 8][bn]) = rb[i];
        } else {
          b[k][lr] = rb[i].x; b[k + 1][lr] = rb[i].y; b[k + 2][lr] = rb[i].z; b[k + 3][lr] = rb[i].w;
        }
      }
    };
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
    __syncthreads();  // (the buffers have been read)
    fetch(kb0);
    put(0);
    __syncthreads();
    for (int kb = kb0; kb < kb1; ++kb) {
      const int buf = (kb - kb0) & 1;
      if (kb + 1 < kb1) fetch(kb + 1);
#pragma unroll
      for (int k = 0; k < RP_K; ++k) {
        const float4 a0 = *reinterpret_cast<const float4*>(&s_a[buf][k][ty]), a1 = *reinterpret_cast<const float4*>(&s_a[buf][k][64 + ty]);
        const float4 b0 = *reinterpret_cast<const float4*>(&s_b[buf][k][tx]), b1 = *reinterpret_cast<const float4*>(&s_b[buf][k][64 + tx]);
        const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          fma2(acc[i][0], acc[i][1], b0.x, b0.y, a[i], a[i]);
          fma2(acc[i][2], acc[i][3], b0.z, b0.w, a[i], a[i]);
          fma2(acc[i][4], acc[i][5], b1.x, b1.y, a[i], a[i]);
          fma2(acc[i][6], acc[i][7], b1.z, b1.w, a[i], a[i]);
        }
      }
      if (kb + 1 < kb1) put(buf ^ 1);
      __syncthreads();
    }
    if (slices > 1) {
      float* mine = p.part + ((size_t)slice * tiles + tile) * (RP_M * RP_N) + tid * 4;  // [sixteen vectors][thread]
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; j += 4)
          *reinterpret_cast<float4*>(mine + (i * 2 + j / 4) * (RP_THREADS * 4)) = make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
      __threadfence();
      __syncthreads();
      if (tid == 0) s_last = atomicAdd(p.part_done + tile, 1) == slices - 1;
      __syncthreads();
      if (!s_last) continue;
      __threadfence();
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
      for (int s = 0; s < slices; ++s) {
        const float* from = p.part + ((size_t)s * tiles + tile) * (RP_M * RP_N) + tid * 4;
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 8; j += 4) {
            const float4 v = __ldcg(reinterpret_cast<const float4*>(from + (i * 2 + j / 4) * (RP_THREADS * 4)));
            acc[i][j] += v.x; acc[i][j + 1] += v.y; acc[i][j + 2] += v.z; acc[i][j + 3] += v.w;
          }
      }
    }
    if (B_BY_K && p.bias != nullptr) {
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        const int n = n0 + (j == 0 ? tx : 64 + tx);
        if (n >= p.N) continue;  // (N % 4 == 0)
        const float4 o = __ldg(reinterpret_cast<const float4*>(p.bias + n));
#pragma unroll
        for (int i = 0; i < 8; ++i) { acc[i][j] += o.x; acc[i][j + 1] += o.y; acc[i][j + 2] += o.z; acc[i][j + 3] += o.w; }
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = m0 + (i < 4 ? ty + i : 60 + ty + i);
      if (r >= n_rows) continue;
      float* dst = p.C + (size_t)row_at(r) * p.N;
#pragma unroll
      for (int j = 0; j < 8; j += 4) {
        const int n = n0 + (j == 0 ? tx : 64 + tx);
        if (p.vec) {
          if (n < p.N) *reinterpret_cast<float4*>(dst + n) = make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (n + q < p.N) dst[n + q] = acc[i][j + q];
        }
      }
    }
  }
}

}  // namespace

int rows_product_launch(RowsProductParams p, bool b_by_k, cudaStream_t stream) {
  const uintptr_t align = reinterpret_cast<uintptr_t>(p.A) | reinterpret_cast<uintptr_t>(p.B) | reinterpret_cast<uintptr_t>(p.part) |
                          reinterpret_cast<uintptr_t>(p.bias);
  if (p.K % 4 != 0 || (b_by_k && p.N % 4 != 0) || (!b_by_k && p.bias != nullptr) || align % 16 != 0 || p.rows == nullptr) return (int)cudaErrorInvalidValue;
  const long long tiles = (long long)((p.max_rows + RP_M - 1) / RP_M) * ((p.N + RP_N - 1) / RP_N);
  if (p.max_rows <= 0) return 0;
  if (tiles > 2147483647LL / 16) return (int)cudaErrorInvalidValue;
  p.vec = p.N % 4 == 0 && reinterpret_cast<uintptr_t>(p.C) % 16 == 0;
  if (b_by_k) launch(rows_product_kernel<true>, RP_SLOTS, RP_THREADS, 0, stream, p);
  else launch(rows_product_kernel<false>, RP_SLOTS, RP_THREADS, 0, stream, p);
  return (int)cudaGetLastError();
}

}  // namespace lmsae
