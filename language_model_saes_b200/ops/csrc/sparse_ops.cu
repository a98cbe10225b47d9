// Sparse decoder forward / backward and the fused gradient + Adam update (sm_100a, plain SIMT kernels:
// these ops are gather- and HBM-bound, not tensor-core work).
//
// Layouts: W_D and W_E^T are both stored feature-major [F, d] (row f contiguous), with an fp32 master
// copy and a bf16 shadow used by the forward kernels. Sparse codes are [B, k] (idx int32, -1 = empty).
//
//  sparse_decode_kernel   x_hat[b,:] = sum_j val[b,j] * W[idx[b,j],:] (+ bias); optional fused MSE loss,
//                         d(x_hat) and d(val) (decoder math of models/sae.py:347-377, loss of
//                         models/sparse_dictionary.py:880-886, gather-GEMM of kernels/kernels.py:383-436
//                         in the reference project)
//  sparse_dact_kernel     d val[b,j] = d x_hat[b,:] . W[idx[b,j],:]           (kernels/kernels.py:327-379)
//  csc_* kernels          group the (row, slot) pairs by feature (counting sort)
//  sparse_grad_adam_kernel  for every feature row f: rebuild dW_D[f,:] = sum act * d x_hat[b,:] and
//                         dW_E^T[f,:] = sum d h * x[b,:] in registers from the feature's entry list and
//                         apply Adam to both rows in the same pass -- the dense gradient is never written
//                         (replaces kernels/kernels.py:137-225 + torch.optim.Adam in the reference).
#include <algorithm>
#include "adam.cuh"
#include "comm_common.cuh"
#include "gather.cuh"

namespace lmsae {

LMSAE_DEFINE_BOUNDS_FETCH(bounds_fetch_sparse_ops)

// ---------------------------------------------------------------------------------------------
// decode (+ loss, + dact)
// ---------------------------------------------------------------------------------------------
// Bound by the gather of B * k decoder rows from L2 / HBM. The unit of work is one WARP per (row, segment of 32 * VPT * 8
// columns), with no barrier and no shared memory on the way: a CTA per row left most of its 512 threads without columns
// below d = 4096 and fetched one decoder row at a time. Warps hold eight row loads in flight each whatever the width.
// VPT = 2 (two 16-byte chunks of every row per lane) from 1024 columns on, where it halves the per-entry bookkeeping
// and still leaves two or more segments per row. Decode + loss of 4096 tokens, before -> now (the code gradients, which the
// first figures include, took about half of it): d 768, k 50: 345 -> 39 us; d 2048, k 128: 1176 -> 170 us (12.6 TB/s of rows out
// of the L2 cache); d 4096, k 50 of a 1.1 GB matrix: 856 -> 242 us (6.9 TB/s).
constexpr int DEC_WARPS = 8;

template <int VPT>
__global__ void __launch_bounds__(DEC_WARPS * 32)
sparse_decode_kernel(const DecodeParams p, int nseg) {
  pdl_wait();
  __shared__ float s_red[DEC_WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = p.d / 8;  // d % 8 == 0
  const long long item = (long long)blockIdx.x * DEC_WARPS + warp;
  const int row = (int)(item / nseg), seg = (int)(item - (long long)row * nseg);
  float local_sq = 0.0f;
  if (row < p.B) {
    int v[VPT];
    bool in[VPT];
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      v[u] = (seg * VPT + u) * 32 + lane;
      in[u] = v[u] < nvec;
    }
    float acc[VPT][8];
    gather_rows_warp<VPT>(p.idx + (size_t)row * p.k, p.val + (size_t)row * p.k, p.k, p.W, p.d, p.F, 1LL << 31, v, in, acc);

    const float rw = (p.row_weight != nullptr) ? p.row_weight[row] : 1.0f;
#pragma unroll
    for (int u = 0; u < VPT; ++u) {
      if (!in[u]) continue;
      const int c = v[u] * 8;
      if (p.bias != nullptr) {
        if ((reinterpret_cast<uintptr_t>(p.bias) & 15) == 0) {
          const float4 b0 = __ldg(reinterpret_cast<const float4*>(p.bias + c)), b1 = __ldg(reinterpret_cast<const float4*>(p.bias + c) + 1);
          acc[u][0] += b0.x; acc[u][1] += b0.y; acc[u][2] += b0.z; acc[u][3] += b0.w;
          acc[u][4] += b1.x; acc[u][5] += b1.y; acc[u][6] += b1.z; acc[u][7] += b1.w;
        } else {  // (a piece of a longer parameter vector starts anywhere)
#pragma unroll
          for (int i = 0; i < 8; ++i) acc[u][i] += __ldg(p.bias + c + i);
        }
      }
      if (p.xhat_f32 != nullptr) {
        float4* o = reinterpret_cast<float4*>(p.xhat_f32 + (size_t)row * p.d + c);
        o[0] = make_float4(acc[u][0], acc[u][1], acc[u][2], acc[u][3]);
        o[1] = make_float4(acc[u][4], acc[u][5], acc[u][6], acc[u][7]);
      }
      if (p.xhat_bf16 != nullptr) {
        uint4 o;
        o.x = pack_bf16x2(acc[u][0], acc[u][1]);
        o.y = pack_bf16x2(acc[u][2], acc[u][3]);
        o.z = pack_bf16x2(acc[u][4], acc[u][5]);
        o.w = pack_bf16x2(acc[u][6], acc[u][7]);
        *reinterpret_cast<uint4*>(p.xhat_bf16 + (size_t)row * p.d + c) = o;
      }
      if (p.label != nullptr) {
        float y[8];
        bf16x8_to_float(__ldg(reinterpret_cast<const uint4*>(p.label + (size_t)row * p.d) + v[u]), y);
        float e[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          e[i] = acc[u][i] - y[i];
          local_sq = fmaf(e[i], e[i], local_sq);
          e[i] *= p.grad_scale * rw;
        }
        uint4 o;
        o.x = pack_bf16x2(e[0], e[1]);
        o.y = pack_bf16x2(e[2], e[3]);
        o.z = pack_bf16x2(e[4], e[5]);
        o.w = pack_bf16x2(e[6], e[7]);
        *reinterpret_cast<uint4*>(p.dxhat + (size_t)row * p.d + c) = o;
      }
    }
    if (p.label != nullptr) {
      local_sq = warp_sum(local_sq);
      if (lane == 0 && p.row_loss != nullptr) p.row_part[item] = local_sq;
      local_sq *= rw;
    }
  }
  if (p.label != nullptr) {
    if (lane == 0) s_red[warp] = local_sq;
    __syncthreads();
    if (warp == 0) {
      float t = lane < DEC_WARPS ? s_red[lane] : 0.0f;
      t = warp_sum(t);
      if (lane == 0) atomicAdd(p.loss_sum, t);
    }
  }
}

// The segments' losses of a row added up in order: the same sum every time.
__global__ void __launch_bounds__(256)
row_loss_kernel(const float* __restrict__ part, int B, int nseg, float* __restrict__ row_loss) {
  pdl_wait();
  const int row = blockIdx.x * 256 + threadIdx.x;
  if (row >= B) return;
  float s = 0.0f;
  for (int i = 0; i < nseg; ++i) s += part[(size_t)row * nseg + i];
  row_loss[row] = s;
}

// A step's loss and the status word to mapped host memory: five floats (the codes are small integers). Two copies and a conversion on the stream, with
// the gaps around them, held the next step up by 24 us.
__global__ void __launch_bounds__(32)
read_back_kernel(const float* __restrict__ loss, const int* __restrict__ status, volatile float* __restrict__ host) {
  pdl_wait();
  if (threadIdx.x < 5) host[threadIdx.x] = threadIdx.x == 0 ? *loss : status != nullptr ? (float)status[threadIdx.x - 1] : 0.0f;
  __threadfence_system();
}

int read_back_launch(const float* loss, const int* status, float* host, cudaStream_t stream) {
  return (int)launch(read_back_kernel, 1, 32, 0, stream, loss, status, host);
}

static int decode_vpt(int d) { return d >= 1024 ? 2 : 1; }
int sparse_decode_segments(int d) { return (d / 8 + 32 * decode_vpt(d) - 1) / (32 * decode_vpt(d)); }

int sparse_decode_launch(const DecodeParams& p, cudaStream_t stream) {
  if (p.d % 8 != 0 || p.d > 8192) return (int)cudaErrorInvalidValue;
  if (p.B <= 0) return 0;
  const int vpt = decode_vpt(p.d), nseg = sparse_decode_segments(p.d);
  const long long blocks = ((long long)p.B * nseg + DEC_WARPS - 1) / DEC_WARPS;
  if (blocks > 2147483647LL) return (int)cudaErrorInvalidValue;
  if (vpt == 2) launch(sparse_decode_kernel<2>, (int)blocks, DEC_WARPS * 32, 0, stream, p, nseg);
  else launch(sparse_decode_kernel<1>, (int)blocks, DEC_WARPS * 32, 0, stream, p, nseg);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && p.label != nullptr && p.row_loss != nullptr) {
    launch(row_loss_kernel, (p.B + 255) / 256, 256, 0, stream, p.row_part, p.B, nseg, p.row_loss);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess || p.label == nullptr || p.dval == nullptr) return (int)e;
  // the code gradients need the whole row's d x_hat: a pass of their own over the same decoder rows
  return sparse_dact_launch(p.idx, p.B, p.k, p.d, p.F, p.W, p.dxhat, p.dval, nullptr, 0, nullptr, stream);
}

// ---------------------------------------------------------------------------------------------
// d val[b,j] = d x_hat[b,:] . W[idx[b,j],:]    (stand-alone, for the feature-sharded path where
// d x_hat only exists after the cross-shard reduction)
// ---------------------------------------------------------------------------------------------
constexpr int DACT_THREADS = 256;

// `wait_pt.world > 0`: d x_hat is the gradient buffer of the fused feature-sharded step, filled by the row owners'
// peer stores; the kernel then waits (bounded) for every owner's flag of `epoch` itself instead of relying on a
// separate wait launch before it.
__global__ void __launch_bounds__(DACT_THREADS)
sparse_dact_kernel(const int* __restrict__ idx, int B, int k, int d, int F, const __nv_bfloat16* __restrict__ W,
                   const __nv_bfloat16* dxhat /* may be peer-written: no read-only path */, float* __restrict__ dval, const PeerTable wait_pt,
                   uint32_t epoch, int* status) {
  pdl_wait();
  extern __shared__ float s_dx[];  // [d]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nvec = d / 8;
  if (wait_pt.world > 0 && !wait_all_sources(wait_pt, kPhaseDxhat, epoch, status)) {
    // the gradient rows never arrived: leave zeros so that nothing downstream consumes stale data
    for (long long i = blockIdx.x * (long long)DACT_THREADS + threadIdx.x; i < (long long)B * k;
         i += (long long)gridDim.x * DACT_THREADS)
      dval[i] = 0.0f;
    return;
  }
  for (int row = blockIdx.x; row < B; row += gridDim.x) {
    __syncthreads();
    for (int v = threadIdx.x; v < nvec; v += DACT_THREADS) {
      float f[8];
      bf16x8_to_float(*(reinterpret_cast<const uint4*>(dxhat + (size_t)row * d) + v), f);
#pragma unroll
      for (int i = 0; i < 8; ++i) s_dx[v * 8 + i] = f[i];
    }
    __syncthreads();
    for (int j = warp; j < k; j += DACT_THREADS / 32) {
      const int f = idx[(size_t)row * k + j];
      float dot = 0.0f;
      if (f >= 0) {
        const uint4* wrow = reinterpret_cast<const uint4*>(W + (size_t)LMSAE_IDX(f, F) * d);
#pragma unroll 4
        for (int v = lane; v < nvec; v += 32) {
          float w[8];
          bf16x8_to_float(__ldg(wrow + v), w);
          const float* dx = s_dx + v * 8;
#pragma unroll
          for (int i = 0; i < 8; ++i) dot = fmaf(w[i], dx[i], dot);
        }
      }
      dot = warp_sum(dot);
      if (lane == 0) dval[(size_t)row * k + j] = dot;
    }
  }
}

int sparse_dact_launch(const int* idx, int B, int k, int d, int F, const __nv_bfloat16* W, const __nv_bfloat16* dxhat,
                       float* dval, const PeerTable* wait, uint32_t epoch, int* status, cudaStream_t stream) {
  if (d % 8 != 0 || (size_t)d * 4 > 160 * 1024) return (int)cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(sparse_dact_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);
  if (e != cudaSuccess) return (int)e;
  int blocks = B < 148 * 8 ? B : 148 * 8;
  PeerTable pt{};
  if (wait != nullptr) pt = *wait;
  launch(sparse_dact_kernel, blocks, DACT_THREADS, (size_t)d * 4, stream, idx, B, k, d, F, W, dxhat, dval, pt, epoch, status);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// MSE loss + gradient on dense rows (feature-sharded path: x_hat arrives from the cross-shard reduce)
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
mse_loss_grad_kernel(const float* __restrict__ xhat, const __nv_bfloat16* __restrict__ label,
                     const float* __restrict__ bias, const float* __restrict__ row_weight, int rows, int d,
                     float grad_scale, __nv_bfloat16* __restrict__ dxhat, float* __restrict__ loss_sum,
                     float* __restrict__ row_loss) {
  pdl_wait();
  __shared__ float s_red[8];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const float rw = row_weight != nullptr ? row_weight[row] : 1.0f;
    float sq = 0.0f;
    for (int c = threadIdx.x; c < d; c += 256) {
      float xh = xhat[(size_t)row * d + c];
      if (bias != nullptr) xh += bias[c];
      const float e = xh - __bfloat162float(label[(size_t)row * d + c]);
      sq = fmaf(e, e, sq);
      dxhat[(size_t)row * d + c] = __float2bfloat16(e * grad_scale * rw);
    }
    sq = warp_sum(sq);
    __syncthreads();
    if (lane == 0) s_red[warp] = sq;
    __syncthreads();
    if (warp == 0) {
      float t = lane < 8 ? s_red[lane] : 0.0f;
      t = warp_sum(t);
      if (lane == 0) {
        if (row_loss != nullptr) row_loss[row] = t;
        atomicAdd(loss_sum, t * rw);
      }
    }
  }
}

int mse_loss_grad_launch(const float* xhat, const __nv_bfloat16* label, const float* bias, const float* row_weight,
                         int rows, int d, float grad_scale, __nv_bfloat16* dxhat, float* loss_sum, float* row_loss,
                         cudaStream_t stream) {
  int blocks = rows < 148 * 8 ? rows : 148 * 8;
  launch(mse_loss_grad_kernel, blocks, 256, 0, stream, xhat, label, bias, row_weight, rows, d, grad_scale, dxhat,
                                                   loss_sum, row_loss);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// Aux-K: losses and gradients of   l = |e|^2 + alpha |e - e_aux|^2   per row, with e = label - x_hat (x_hat from
// the main codes) and e_aux the reconstruction of the residual from dead features
// (models/sparse_dictionary.py:941-991 of the reference project; e is NOT detached there, so the auxiliary term
// also pulls on x_hat). Outputs, per row scaled by grad_scale * row_weight:
//   g_main = d l / d x_hat = (x_hat - label) - alpha * r,      g_aux = d l / d e_aux = -alpha * r,   r = e - e_aux
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
auxk_loss_grad_kernel(const float* __restrict__ xhat, const float* __restrict__ aux_rec,
                      const __nv_bfloat16* __restrict__ label, const float* __restrict__ bias,
                      const float* __restrict__ row_weight, int rows, int d, float grad_scale, float alpha_host,
                      const float* __restrict__ alpha_factor, __nv_bfloat16* __restrict__ g_main,
                      __nv_bfloat16* __restrict__ g_aux, float* __restrict__ loss_sum, float* __restrict__ aux_sum) {
  pdl_wait();
  __shared__ float s_red[2][8];
  // alpha_factor (one device float, optional): 0 switches the auxiliary term off without the host knowing, e.g. in a step
  // that has no dead feature
  const float alpha = alpha_factor != nullptr ? alpha_host * *alpha_factor : alpha_host;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int row = blockIdx.x; row < rows; row += gridDim.x) {
    const float rw = row_weight != nullptr ? row_weight[row] : 1.0f;
    const float sc = grad_scale * rw;
    float sq = 0.0f, sq_aux = 0.0f;
    for (int c = threadIdx.x; c < d; c += 256) {
      const size_t o = (size_t)row * d + c;
      float xh = xhat[o];
      if (bias != nullptr) xh += bias[c];
      const float e = __bfloat162float(label[o]) - xh;
      const float r = e - aux_rec[o];
      sq = fmaf(e, e, sq);
      sq_aux = fmaf(r, r, sq_aux);
      g_main[o] = __float2bfloat16(-(e + alpha * r) * sc);
      g_aux[o] = __float2bfloat16(-alpha * r * sc);
    }
    sq = warp_sum(sq);
    sq_aux = warp_sum(sq_aux);
    __syncthreads();
    if (lane == 0) { s_red[0][warp] = sq; s_red[1][warp] = sq_aux; }
    __syncthreads();
    if (warp == 0) {
      float t = lane < 8 ? s_red[0][lane] : 0.0f, u = lane < 8 ? s_red[1][lane] : 0.0f;
      t = warp_sum(t);
      u = warp_sum(u);
      if (lane == 0) {
        atomicAdd(loss_sum, t * rw);
        atomicAdd(aux_sum, alpha * u * rw);
      }
    }
  }
}

int auxk_loss_grad_launch(const float* xhat, const float* aux_rec, const __nv_bfloat16* label, const float* bias,
                          const float* row_weight, int rows, int d, float grad_scale, float alpha,
                          const float* alpha_factor, __nv_bfloat16* g_main, __nv_bfloat16* g_aux, float* loss_sum,
                          float* aux_sum, cudaStream_t stream) {
  int blocks = rows < 148 * 8 ? rows : 148 * 8;
  if (blocks <= 0) return 0;
  launch(auxk_loss_grad_kernel, blocks, 256, 0, stream, xhat, aux_rec, label, bias, row_weight, rows, d, grad_scale, alpha,
                                                    alpha_factor, g_main, g_aux, loss_sum, aux_sum);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// group (row, slot) pairs by feature: counts -> offsets (exclusive scan) -> entries
// ---------------------------------------------------------------------------------------------
// (A kernel, because a fill on the stream cannot be launched ahead: 2 us with the gaps around it.)
__global__ void csc_zero_kernel(int* __restrict__ counts, int F, int* __restrict__ heavy) {
  pdl_wait();
  if (heavy != nullptr && blockIdx.x == 0 && threadIdx.x == 0) heavy[0] = 0;  // (counted by the scan)
  const int i0 = (blockIdx.x * blockDim.x + threadIdx.x) * 4;
  if (i0 + 3 < F && reinterpret_cast<uintptr_t>(counts) % 16 == 0) {
    *reinterpret_cast<int4*>(counts + i0) = make_int4(0, 0, 0, 0);
  } else {
    for (int i = i0; i < min(i0 + 4, F); ++i) counts[i] = 0;
  }
}

__global__ void csc_count_kernel(const int* __restrict__ idx, long long n, int F, int* __restrict__ counts) {
  pdl_wait();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int f = idx[i];
    if (f >= 0 && f < F) atomicAdd(&counts[f], 1);
  }
}

// Exclusive scan of counts[F] in three small launches: per-block scan of 4096 elements (coalesced int4
// loads) + block totals, scan of the totals by one block, then add-back while writing offsets and cursors.
constexpr int SCAN_THREADS = 1024;
constexpr int SCAN_ELEMS = SCAN_THREADS * 4;

__device__ __forceinline__ int block_exclusive_scan_1024(int v, int* s_warp, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    int w = s_warp[lane];
    int winc = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, winc, o);
      if (lane >= o) winc += t;
    }
    s_warp[lane] = winc - w;  // exclusive prefix of the warp totals
    if (lane == 31) s_warp[32] = winc;
  }
  __syncthreads();
  total = s_warp[32];
  return s_warp[warp] + inc - v;
}

__global__ void __launch_bounds__(SCAN_THREADS)
csc_scan_local_kernel(const int* __restrict__ counts, int F, int* __restrict__ offsets, int* __restrict__ block_sums,
                      int* __restrict__ heavy, int heavy_cap) {
  pdl_wait();
  __shared__ int s_warp[33];
  const int base = blockIdx.x * SCAN_ELEMS + threadIdx.x * 4;
  int c[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    c[i] = (base + i < F) ? counts[base + i] : 0;
    if (heavy != nullptr && c[i] > kHeavyRow) {
      const int pos = atomicAdd(heavy, 1);
      if (pos < heavy_cap) heavy[1 + pos] = base + i;
    }
  }
  const int mine = c[0] + c[1] + c[2] + c[3];
  int total;
  int run = block_exclusive_scan_1024(mine, s_warp, total);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (base + i < F) offsets[base + i] = run;
    run += c[i];
  }
  if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

__global__ void __launch_bounds__(SCAN_THREADS)
csc_scan_sums_kernel(int* __restrict__ block_sums, int nblocks, int* __restrict__ offsets, int F) {
  pdl_wait();
  __shared__ int s_warp[33];
  __shared__ int s_carry;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (int b0 = 0; b0 < nblocks; b0 += SCAN_THREADS) {
    const int i = b0 + threadIdx.x;
    const int v = i < nblocks ? block_sums[i] : 0;
    int total;
    const int ex = block_exclusive_scan_1024(v, s_warp, total);
    const int carry = s_carry;
    if (i < nblocks) block_sums[i] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) s_carry = carry + total;
    __syncthreads();
  }
  if (threadIdx.x == 0) offsets[F] = s_carry;
}

__global__ void __launch_bounds__(SCAN_THREADS)
csc_scan_add_kernel(const int* __restrict__ block_sums, int F, int* __restrict__ offsets, int* __restrict__ cursor) {
  pdl_wait();
  const int add = block_sums[blockIdx.x];
  const int base = blockIdx.x * SCAN_ELEMS + threadIdx.x * 4;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (base + i < F) {
      const int o = offsets[base + i] + add;
      offsets[base + i] = o;
      if (cursor != nullptr) cursor[base + i] = o;
    }
  }
}

// The three in one launch: a block adds up all counts before its own 4096 instead of waiting for the other blocks' totals. The last block
// reads the whole array from L2: up to 2^17 features (half a megabyte, 4 us) that costs less than two launches (24576 features: 9.1 ->
// 6.0 us, and a memset less).
constexpr int kOneScanFeatures = 1 << 17;
__global__ void __launch_bounds__(SCAN_THREADS)
csc_scan_kernel(const int* __restrict__ counts, int F, int* __restrict__ offsets, int* __restrict__ cursor, int* __restrict__ heavy, int heavy_cap) {
  pdl_wait();
  __shared__ int s_warp[33];
  const int first = blockIdx.x * SCAN_ELEMS, base = first + threadIdx.x * 4;
  int before = 0;
#pragma unroll 4
  for (int i = threadIdx.x; i < first / 4; i += SCAN_THREADS) {
    const int4 c = __ldg(reinterpret_cast<const int4*>(counts) + i);
    before += c.x + c.y + c.z + c.w;
  }
  int carry;
  block_exclusive_scan_1024(before, s_warp, carry);
  __syncthreads();  // (the scan's words are used again)
  int c[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    c[i] = (base + i < F) ? counts[base + i] : 0;
    if (heavy != nullptr && c[i] > kHeavyRow) {
      const int pos = atomicAdd(heavy, 1);
      if (pos < heavy_cap) heavy[1 + pos] = base + i;
    }
  }
  int total;
  int run = carry + block_exclusive_scan_1024(c[0] + c[1] + c[2] + c[3], s_warp, total);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if (base + i < F) {
      offsets[base + i] = run;
      cursor[base + i] = run;
    }
    run += c[i];
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) offsets[F] = carry + total;
}

__global__ void csc_fill_kernel(const int* __restrict__ idx, long long n, int F, int* __restrict__ cursor,
                                int* __restrict__ entries) {
  pdl_wait();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int f = idx[i];
    if (f >= 0 && f < F) {
      const int pos = atomicAdd(&cursor[f], 1);
      entries[pos] = (int)i;
    }
  }
}

// All of it in one launch, and no block waits for another: a block owns `span` features and reads all entries, keeps those of its features in lists in
// shared memory (one per warp, feature and position in one word) and counts the entries of features before its own, which is where its offsets begin.
// Counts, their scan and the places of the entries then come from the lists. Bound by the instructions of the reading (a subtraction with borrow, a
// comparison and a ballot per entry in every block), so for few entries. Against a fill and three launches: 4096 entries of 256 features 10.3 -> 4.1 us,
// 32768 of 4096 9.4 -> 6.7 (with three features in every row 11.2 -> 9.1), 512 of 131072 11.9 -> 4.4; at 111037 entries it would be 12.8 -> 13.2. The line
// lies where a warp's list holds all that the warp reads, so that no list overflows. Lists per thread without ballots (6.7 -> 6.9), the next
// entries fetched ahead (7.3) and places drawn by lanes of one feature together (8.1) were slower at 32768.
// `places` counts the long rows, a word of its own that is zero between calls: the blocks take their places in the list `heavy` from its low bits,
// and the one that finds all others counted in its high bits leaves the number in heavy[0] and the zero.
constexpr int kRangeBlocks = 148, kRangeSpan = 1 << 12, kRangeTile = SCAN_THREADS * 4, kRangeTiles = 11;
__global__ void __launch_bounds__(SCAN_THREADS, 1)
csc_ranges_kernel(const int* __restrict__ idx, int n, int F, int span, int cap, int* __restrict__ counts, int* __restrict__ offsets,
                  int* __restrict__ cursor, int* __restrict__ entries, int* __restrict__ heavy, int* __restrict__ places) {
  pdl_wait();
  extern __shared__ int s_cnt[];  // [span]: counts, then cursors; then the lists
  __shared__ int s_warp[33];
  __shared__ int s_heavy, s_heavy_at;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned* const list = reinterpret_cast<unsigned*>(s_cnt + span) + warp * cap;
  const int lo = blockIdx.x * span, width = min(span, F - lo);
  for (int i = threadIdx.x; i < span; i += SCAN_THREADS) s_cnt[i] = 0;
  if (threadIdx.x == 0) s_heavy = 0;

  constexpr int U = 4;
  int before = 0, mine = 0;
  for (int i0 = warp * 128; i0 < n; i0 += kRangeTile * U) {
    int4 f[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * kRangeTile + lane * 4;
      f[u] = make_int4(-1, -1, -1, -1);
      if (i + 3 < n) {
        f[u] = __ldg(reinterpret_cast<const int4*>(idx + i));
      } else if (i < n) {
        f[u].x = idx[i];
        if (i + 1 < n) f[u].y = idx[i + 1];
        if (i + 2 < n) f[u].z = idx[i + 2];
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int i = i0 + u * kRangeTile;
      if (i >= n) break;
      const int v[4] = {f[u].x, f[u].y, f[u].z, f[u].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        unsigned rel;
        asm("sub.cc.u32 %0, %2, %3;\n\tsubc.u32 %1, %1, 0;" : "=r"(rel), "+r"(before) : "r"(v[j]), "r"(lo));  // (before: less one for an entry below lo)
        const bool in = rel < (unsigned)width;
        const unsigned m = __ballot_sync(0xffffffffu, in);
        if (m != 0) {
          if (in) list[LMSAE_IDX(mine + __popc(m & ((1u << lane) - 1)), cap)] = rel << 20 | (unsigned)(i + lane * 4 + j);
          mine += __popc(m);
        }
      }
    }
  }
  int carry;
  block_exclusive_scan_1024(-before, s_warp, carry);  // (its barriers: the counts are zero)
  for (int e = lane; e < mine; e += 32) atomicAdd(&s_cnt[list[e] >> 20], 1);
  __syncthreads();
  int c[4], place[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rel = threadIdx.x * 4 + i;
    c[i] = rel < width ? s_cnt[rel] : 0;
    place[i] = heavy != nullptr && c[i] > kHeavyRow ? atomicAdd(&s_heavy, 1) : -1;
  }
  int total;
  int run = carry + block_exclusive_scan_1024(c[0] + c[1] + c[2] + c[3], s_warp, total);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rel = threadIdx.x * 4 + i;
    if (rel < width) {
      counts[lo + rel] = c[i];
      offsets[lo + rel] = run;
      s_cnt[rel] = run;
      cursor[lo + rel] = run + c[i];
    }
    run += c[i];
  }
  if (threadIdx.x == 0) {
    if (lo + width == F) offsets[F] = carry + total;
    if (heavy != nullptr) {
      const unsigned before_me = atomicAdd(reinterpret_cast<unsigned*>(places), (1u << 24) + (unsigned)s_heavy);
      s_heavy_at = (int)(before_me & 0xffffffu);
      if ((before_me >> 24) == gridDim.x - 1) {
        heavy[0] = s_heavy_at + s_heavy;
        *places = 0;
      }
    }
  }
  __syncthreads();
  for (int e = lane; e < mine; e += 32) entries[LMSAE_IDX(atomicAdd(&s_cnt[list[e] >> 20], 1), n)] = (int)(list[e] & 0xfffffu);
#pragma unroll
  for (int i = 0; i < 4; ++i)
    if (place[i] >= 0) heavy[1 + s_heavy_at + place[i]] = lo + threadIdx.x * 4 + i;
}

int csc_build_launch(const int* idx, long long n, int F, int* counts, int* offsets, int* cursor, int* entries,
                     int* block_sums_buf, int* heavy, int heavy_cap, int* places, cudaStream_t stream) {
  if (n < 0 || n > 2147483647LL || F <= 0) return (int)cudaErrorInvalidValue;  // positions are stored as 32-bit ints
  if (heavy != nullptr && (long long)heavy_cap < n / (kHeavyRow + 1)) return (int)cudaErrorInvalidValue;  // room for every row there can be
  if (n <= kRangeTiles * kRangeTile && F <= kRangeBlocks * kRangeSpan && reinterpret_cast<uintptr_t>(idx) % 16 == 0 && (heavy == nullptr || places != nullptr)) {
    const int span = std::max(32, ((F + kRangeBlocks - 1) / kRangeBlocks + 3) & ~3);
    const int cap = (int)((n + kRangeTile - 1) / kRangeTile) * 128;
    const int smem = (int)sizeof(int) * (span + cap * (SCAN_THREADS / 32));
    const cudaError_t e = cudaFuncSetAttribute(csc_ranges_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)sizeof(int) * (kRangeSpan + kRangeTiles * 128 * (SCAN_THREADS / 32)));
    if (e != cudaSuccess) return (int)e;
    return (int)launch(csc_ranges_kernel, (F + span - 1) / span, SCAN_THREADS, smem, stream, idx, (int)n, F, span, cap, counts, offsets, cursor, entries, heavy,
                       places);
  }
  launch(csc_zero_kernel, (int)(((long long)F + 1023) / 1024), 256, 0, stream, counts, F, heavy);
  const int threads = 256;
  int blocks = (int)((n + threads - 1) / threads);
  if (blocks > 148 * 8) blocks = 148 * 8;
  if (blocks < 1) blocks = 1;
  launch(csc_count_kernel, blocks, threads, 0, stream, idx, n, F, counts);
  // `block_sums_buf` holds one int per 4096 features
  const int nblocks = (F + SCAN_ELEMS - 1) / SCAN_ELEMS;
  if (F <= kOneScanFeatures && reinterpret_cast<uintptr_t>(counts) % 16 == 0) {
    launch(csc_scan_kernel, nblocks, SCAN_THREADS, 0, stream, counts, F, offsets, cursor, heavy, heavy_cap);
  } else {
    int* block_sums = block_sums_buf;
    launch(csc_scan_local_kernel, nblocks, SCAN_THREADS, 0, stream, counts, F, offsets, block_sums, heavy, heavy_cap);
    launch(csc_scan_sums_kernel, 1, SCAN_THREADS, 0, stream, block_sums, nblocks, offsets, F);
    launch(csc_scan_add_kernel, nblocks, SCAN_THREADS, 0, stream, block_sums, F, offsets, cursor);
  }
  launch(csc_fill_kernel, blocks, threads, 0, stream, idx, n, F, cursor, entries);
  return (int)cudaGetLastError();
}

// offsets[0..n] = exclusive prefix sum of counts[0..n-1] (offsets[n] = total); `block_sums_buf`: one int per 4096 counts
int exclusive_scan_launch(const int* counts, int n, int* offsets, int* block_sums_buf, cudaStream_t stream) {
  if (n <= 0) return (int)cudaErrorInvalidValue;
  const int nblocks = (n + SCAN_ELEMS - 1) / SCAN_ELEMS;
  launch(csc_scan_local_kernel, nblocks, SCAN_THREADS, 0, stream, counts, n, offsets, block_sums_buf, nullptr, 0);
  launch(csc_scan_sums_kernel, 1, SCAN_THREADS, 0, stream, block_sums_buf, nblocks, offsets, n);
  launch(csc_scan_add_kernel, nblocks, SCAN_THREADS, 0, stream, block_sums_buf, n, offsets, nullptr);
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// fused sparse gradient + Adam over feature rows
// ---------------------------------------------------------------------------------------------


constexpr int GA_THREADS = 256;

__device__ __forceinline__ float4 ldcs4(const float* p) { return __ldcs(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ void stcs4(float* p, const float4& v) { __stcs(reinterpret_cast<float4*>(p), v); }

// One CTA walks feature rows (grid-stride). For a row it first rebuilds the two gradient rows from the
// feature's entry list (gathers of x / d x_hat rows, normally L2 hits), then streams p, m, v once.
// VEC = float4 groups per thread and chunk step. VEC 1 with four CTAs per SM is the stand-alone form (most warps to
// hide latency). VEC 2 with two CTAs per SM keeps the same number of bytes in flight per SM (twelve 16-byte loads per
// thread) with half the warps and registers-per-SM to spare: the form that shares the SMs with a concurrently running
// encoder GEMM of the next step.
// SIDES: 3 = both matrices, 1 = decoder side only, 2 = encoder side only (compile-time, so a one-sided launch carries no
// registers for the other side). One-sided launches serve dictionaries with short rows and several decoder matrices per
// encoder (cross-layer transcoders): a row is then one chunk, and what bounds the kernel is the chain offsets -> entries
// -> codes -> gathered rows -> parameters per row. There the parameter and moment loads are issued BEFORE the entry loop
// (EARLY), so that their trip to HBM overlaps the gathers, which mostly hit L2.
template <int VEC, int MIN_CTAS, int SIDES>
__global__ void __launch_bounds__(GA_THREADS, MIN_CTAS)
sparse_grad_adam_kernel(const GradAdamParams p) {
  constexpr bool doD = (SIDES & 1) != 0, doE = (SIDES & 2) != 0;
  constexpr bool EARLY = SIDES != 3;
  __shared__ float s_red[GA_THREADS / 32];
  __shared__ float s_gsq[GA_THREADS / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const float gmul = p.grad_mul != nullptr ? *p.grad_mul : 1.0f;
  float gsq_local = 0.0f;
  // An earlier kernel of this step gave up on a bounded wait (its inputs never arrived): the codes and gradient rows
  // this kernel would consume are stale, so the parameters and moments stay as they are until the host has seen the
  // status word.
  const bool skip = p.status != nullptr && *reinterpret_cast<const volatile int*>(p.status) != 0;

  for (int f = p.f_begin + blockIdx.x; f < p.f_end && !skip; f += gridDim.x) {
    const int e0 = p.offsets[f], e1 = p.offsets[f + 1];
    const int xr = p.extra_row != nullptr ? p.extra_row[f] : -1;
    const float self_scale = p.wd_self_scale != nullptr ? p.wd_self_scale[f] * gmul : 0.0f;
    float bias_g = (xr >= 0 && p.extra_gb != nullptr) ? p.extra_gb[xr] : 0.0f;
    float norm_sq = 0.0f;
    for (int c0 = 0; c0 < p.d; c0 += GA_THREADS * 4 * VEC) {
      int c[VEC];
      bool in[VEC];
      size_t o[VEC], os[VEC];
      float gD[VEC][4], gE[VEC][4];
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        c[v] = c0 + v * GA_THREADS * 4 + threadIdx.x * 4;
        in[v] = c[v] < p.d;  // d % 4 == 0
        o[v] = (size_t)f * p.d + (in[v] ? c[v] : 0);                  // parameters, shadows, dense gradient outputs
        os[v] = (size_t)(f - p.state_f0) * p.d + (in[v] ? c[v] : 0);  // moments
#pragma unroll
        for (int i = 0; i < 4; ++i) gD[v][i] = gE[v][i] = 0.0f;
        if (xr >= 0 && in[v]) {
          if (doD && p.extra_gD != nullptr) {
            const float4 a = *reinterpret_cast<const float4*>(p.extra_gD + (size_t)xr * p.d + c[v]);
            gD[v][0] = a.x; gD[v][1] = a.y; gD[v][2] = a.z; gD[v][3] = a.w;
          }
          if (doE && p.extra_gE != nullptr) {
            const float4 b = *reinterpret_cast<const float4*>(p.extra_gE + (size_t)xr * p.d + c[v]);
            gE[v][0] = b.x; gE[v][1] = b.y; gE[v][2] = b.z; gE[v][3] = b.w;
          }
        }
      }
      float4 w[VEC], m[VEC], vv[VEC], we[VEC], me[VEC], ve[VEC];
      if constexpr (EARLY) {
        if (p.update) {
#pragma unroll
          for (int v = 0; v < VEC; ++v) {
            if (in[v]) {
              if constexpr (doD) { w[v] = ldcs4(p.WD + o[v]); m[v] = ldcs4(p.mD + os[v]); vv[v] = ldcs4(p.vD + os[v]); }
              if constexpr (doE) { we[v] = ldcs4(p.WE + o[v]); me[v] = ldcs4(p.mE + os[v]); ve[v] = ldcs4(p.vE + os[v]); }
            }
          }
        }
      }
      // The entries' metadata (position, token row, code, code gradient) is fetched 32 entries at a time, one entry per
      // lane, and handed round by shuffles: one coalesced load and one integer division per entry and warp instead of
      // three dependent broadcast loads and a division per entry and THREAD, and the row gathers of successive entries
      // no longer wait for index loads in between.
      for (int eb = e0; eb < e1; eb += 32) {
        const int n_e = min(32, e1 - eb);
        int row_l = 0, aux_l = 0;
        float a_l = 0.0f, da_l = 0.0f;
        if (lane < n_e) {
          const int ent = (int)LMSAE_IDX(p.entries[eb + lane], p.n_codes);
          row_l = (int)LMSAE_IDX(ent / p.k, p.n_rows);
          a_l = p.act[ent];
          da_l = p.dact[ent];
          // codes beyond the first k_main slots of a row (auxiliary codes) multiply the auxiliary output gradient
          aux_l = (p.dxhat_aux != nullptr && ent - row_l * p.k >= p.k_main) ? 1 : 0;
        }
        for (int j = 0; j < n_e; ++j) {
          const int row = __shfl_sync(0xffffffffu, row_l, j);
          const float a = __shfl_sync(0xffffffffu, a_l, j);
          const float da = __shfl_sync(0xffffffffu, da_l, j);
          const __nv_bfloat16* gmat = __shfl_sync(0xffffffffu, aux_l, j) ? p.dxhat_aux : p.dxhat;
          if (c0 == 0 && threadIdx.x == 0) bias_g += da;
#pragma unroll
          for (int v = 0; v < VEC; ++v) {
            if (in[v]) {
              if constexpr (doD) {
                const uint2 ud = __ldg(reinterpret_cast<const uint2*>(gmat + (size_t)row * p.d + c[v]));
                const float2 d01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ud.x));
                const float2 d23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ud.y));
                gD[v][0] = fmaf(a, d01.x, gD[v][0]); gD[v][1] = fmaf(a, d01.y, gD[v][1]);
                gD[v][2] = fmaf(a, d23.x, gD[v][2]); gD[v][3] = fmaf(a, d23.y, gD[v][3]);
              }
              if constexpr (doE) {
                const uint2 ux = __ldg(reinterpret_cast<const uint2*>(p.x + (size_t)row * p.d + c[v]));
                const float2 x01 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ux.x));
                const float2 x23 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&ux.y));
                gE[v][0] = fmaf(da, x01.x, gE[v][0]); gE[v][1] = fmaf(da, x01.y, gE[v][1]);
                gE[v][2] = fmaf(da, x23.x, gE[v][2]); gE[v][3] = fmaf(da, x23.y, gE[v][3]);
              }
            }
          }
        }
      }
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        if (!in[v]) continue;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          gD[v][i] *= gmul;
          gE[v][i] *= gmul;
          gsq_local += gD[v][i] * gD[v][i] + gE[v][i] * gE[v][i];
        }
        if (p.gD_out != nullptr) *reinterpret_cast<float4*>(p.gD_out + o[v]) = make_float4(gD[v][0], gD[v][1], gD[v][2], gD[v][3]);
        if (p.gE_out != nullptr) *reinterpret_cast<float4*>(p.gE_out + o[v]) = make_float4(gE[v][0], gE[v][1], gE[v][2], gE[v][3]);
      }
      if (p.update) {
        // all streams of this chunk step are requested before the first is used (96 bytes in flight per thread and VEC)
        if constexpr (!EARLY) {
#pragma unroll
          for (int v = 0; v < VEC; ++v) {
            if (in[v]) {
              if constexpr (doD) { w[v] = ldcs4(p.WD + o[v]); m[v] = ldcs4(p.mD + os[v]); vv[v] = ldcs4(p.vD + os[v]); }
              if constexpr (doE) { we[v] = ldcs4(p.WE + o[v]); me[v] = ldcs4(p.mE + os[v]); ve[v] = ldcs4(p.vE + os[v]); }
            }
          }
        }
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
          if (!in[v]) continue;
          if constexpr (doD) {
            if (self_scale != 0.0f) {  // (not part of the squared-norm accumulation above: a penalty term's share is small)
              gD[v][0] = fmaf(self_scale, w[v].x, gD[v][0]); gD[v][1] = fmaf(self_scale, w[v].y, gD[v][1]);
              gD[v][2] = fmaf(self_scale, w[v].z, gD[v][2]); gD[v][3] = fmaf(self_scale, w[v].w, gD[v][3]);
            }
            adam_elem(w[v].x, m[v].x, vv[v].x, gD[v][0], p.h); adam_elem(w[v].y, m[v].y, vv[v].y, gD[v][1], p.h);
            adam_elem(w[v].z, m[v].z, vv[v].z, gD[v][2], p.h); adam_elem(w[v].w, m[v].w, vv[v].w, gD[v][3], p.h);
            stcs4(p.WD + o[v], w[v]); stcs4(p.mD + os[v], m[v]); stcs4(p.vD + os[v], vv[v]);
            norm_sq += w[v].x * w[v].x + w[v].y * w[v].y + w[v].z * w[v].z + w[v].w * w[v].w;
            uint2 sh; sh.x = pack_bf16x2(w[v].x, w[v].y); sh.y = pack_bf16x2(w[v].z, w[v].w);
            if (SIDES == 3 && p.n_pub > 0) {
              for (int q = 0; q < p.n_pub; ++q)
                *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.pub.base[q] + p.pub_wd_off) + o[v]) = sh;
            } else {
              *reinterpret_cast<uint2*>(p.WD_bf16 + o[v]) = sh;
            }
          }
          if constexpr (doE) {
            adam_elem(we[v].x, me[v].x, ve[v].x, gE[v][0], p.h); adam_elem(we[v].y, me[v].y, ve[v].y, gE[v][1], p.h);
            adam_elem(we[v].z, me[v].z, ve[v].z, gE[v][2], p.h); adam_elem(we[v].w, me[v].w, ve[v].w, gE[v][3], p.h);
            stcs4(p.WE + o[v], we[v]); stcs4(p.mE + os[v], me[v]); stcs4(p.vE + os[v], ve[v]);
            uint2 sh; sh.x = pack_bf16x2(we[v].x, we[v].y); sh.y = pack_bf16x2(we[v].z, we[v].w);
            if (SIDES == 3 && p.n_pub > 0) {
              for (int q = 0; q < p.n_pub; ++q)
                *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.pub.base[q] + p.pub_we_off) + o[v]) = sh;
            } else {
              *reinterpret_cast<uint2*>(p.WE_bf16 + o[v]) = sh;
            }
          }
        }
      }
    }
    if (threadIdx.x == 0) {
      bias_g *= gmul;
      gsq_local += bias_g * bias_g;
      if (p.update && p.bE != nullptr && doE) {
        float b = p.bE[f], m = p.mbE[f - p.state_f0], v = p.vbE[f - p.state_f0];
        adam_elem(b, m, v, bias_g, p.h);
        p.mbE[f - p.state_f0] = m; p.vbE[f - p.state_f0] = v;
        if (SIDES == 3 && p.n_pub > 0) {
          for (int q = 0; q < p.n_pub; ++q) reinterpret_cast<float*>(p.pub.base[q] + p.pub_be_off)[f] = b;
        } else {
          p.bE[f] = b;
        }
      }
    }
    if (p.update && doD && (p.dec_norm != nullptr || p.norm_sq_accum != nullptr)) {
      norm_sq = warp_sum(norm_sq);
      __syncthreads();
      if (lane == 0) s_red[warp] = norm_sq;
      __syncthreads();
      if (warp == 0) {
        float t = lane < GA_THREADS / 32 ? s_red[lane] : 0.0f;
        t = warp_sum(t);
        if (lane == 0) {
          if (p.norm_sq_accum != nullptr) {
            p.norm_sq_accum[f] += t;  // one CTA per row and launch: the squared norms of several matrices add up here
          } else if (SIDES == 3 && p.n_pub > 0) {
            for (int q = 0; q < p.n_pub; ++q) reinterpret_cast<float*>(p.pub.base[q] + p.pub_norm_off)[f] = sqrtf(t);
          } else {
            p.dec_norm[f] = sqrtf(t);
          }
        }
      }
    }
  }
  if (p.grad_sq_sum != nullptr) {
    gsq_local = warp_sum(gsq_local);
    if (lane == 0) s_gsq[warp] = gsq_local;
    __syncthreads();
    if (warp == 0) {
      float t = lane < GA_THREADS / 32 ? s_gsq[lane] : 0.0f;
      t = warp_sum(t);
      if (lane == 0) atomicAdd(p.grad_sq_sum, t);
    }
  }
  // published even when the update was skipped, so that the replicas waiting for this rank's rows do not time out too
  if constexpr (SIDES == 3) {
    if (p.n_pub > 0 && p.update) signal_peers_when_grid_done(p.pub, kPhaseParams, p.pub_epoch, p.pub_done);
  }
}

int sparse_grad_adam_launch(const GradAdamParams& p, cudaStream_t stream) {
  if (p.d % 4 != 0) return (int)cudaErrorInvalidValue;
  const int rows = p.f_end - p.f_begin;
  if (rows <= 0) return 0;
  // CTAs are persistent (grid-stride over feature rows): the grid size sets how many share an SM
  if (p.n_pub < 0 || p.n_pub > kMaxPeers || (p.n_pub > 0 && p.n_pub != p.pub.world)) return (int)cudaErrorInvalidValue;
  if (p.state_f0 < 0 || p.state_f0 > p.f_begin) return (int)cudaErrorInvalidValue;
  const int cap = (p.ctas_per_sm >= 1 && p.ctas_per_sm <= 4) ? 148 * p.ctas_per_sm : 148 * 8;
  int blocks = rows < cap ? rows : cap;
  const bool doD = p.WD != nullptr, doE = p.WE != nullptr;
  if (!doD && !doE) return (int)cudaErrorInvalidValue;
  if (!(doD && doE) && p.n_pub > 0) return (int)cudaErrorInvalidValue;  // rows are published by two-sided launches only
  if (p.layer_rows != 0 && (doD || p.layer_rows < 0 || p.F % p.layer_rows != 0 || !grad_adam_rows_supported(p))) return (int)cudaErrorInvalidValue;
  if (grad_adam_rows_supported(p)) return grad_adam_rows_launch(p, stream);
  if (p.dact_mode != 0) return (int)cudaErrorInvalidValue;  // the kernel below takes the code gradients as an input
  if (doD && doE) {
    if (p.ctas_per_sm >= 1 && p.ctas_per_sm <= 2)
      launch_plain(sparse_grad_adam_kernel<2, 2, 3>, blocks, GA_THREADS, 0, stream, p);
    else
      launch_plain(sparse_grad_adam_kernel<1, 4, 3>, blocks, GA_THREADS, 0, stream, p);
  } else {
    // one-sided: fewer registers; the encoder side fits five CTAs (rows in flight) per SM, the decoder side (row norms,
    // norm penalty) four without spilling
    const int per_sm = doD ? 4 : 5;
    if (p.ctas_per_sm < 1 || p.ctas_per_sm > per_sm) blocks = rows < 148 * per_sm ? rows : 148 * per_sm;
    if (doD) launch_plain(sparse_grad_adam_kernel<1, 4, 1>, blocks, GA_THREADS, 0, stream, p);
    else launch_plain(sparse_grad_adam_kernel<1, 5, 2>, blocks, GA_THREADS, 0, stream, p);
  }
  return (int)cudaGetLastError();
}

// ---------------------------------------------------------------------------------------------
// dense helpers: column sum of a bf16 matrix, and a flat Adam step with an explicit gradient
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
colsum_bf16_kernel(const __nv_bfloat16* __restrict__ a, int rows, int d, int rows_per_block, float* __restrict__ out) {
  pdl_wait();
  const int r0 = blockIdx.y * rows_per_block;
  const int r1 = min(rows, r0 + rows_per_block);
  for (int c = blockIdx.x * 256 + threadIdx.x; c < d; c += gridDim.x * 256) {
    float s = 0.0f;
    for (int r = r0; r < r1; ++r) s += __bfloat162float(a[(size_t)r * d + c]);
    atomicAdd(out + c, s);
  }
}

int colsum_bf16_launch(const __nv_bfloat16* a, int rows, int d, float* out, cudaStream_t stream) {
  cudaError_t e = cudaMemsetAsync(out, 0, (size_t)d * sizeof(float), stream);
  if (e != cudaSuccess) return (int)e;
  const int rows_per_block = 64;
  dim3 grid((d + 255) / 256, (rows + rows_per_block - 1) / rows_per_block);
  launch(colsum_bf16_kernel, grid, 256, 0, stream, a, rows, d, rows_per_block, out);
  return (int)cudaGetLastError();
}

// Decoder (and projection) biases at the end of a step, in one launch: the gradient of a bias is the column sum of a bf16 matrix
// [rows, d]; the same launch applies Adam to it and turns the step's loss sum into the mean, leaving the sum at zero for the next
// step. Several matrices of the same number of rows share a launch.
//   grid (blocks of 256 columns, row blocks): lanes of a warp own eight columns (16-byte loads, four in flight), its eight warps every
//   eighth row; the row blocks' sums go through memory, and the last row block of a column block to arrive adds them up in order
//   (the sum does not depend on the order of arrival) and applies Adam.
// As five launches (fill, column sums by atomics, Adam; a fill and a division for the loss): 4096 rows of 768: 7.7 + 2.8 + 5 us, 4096
// rows of 4096: 14.6 + 2.8 + 5; here 9.6 and 14.8. In steps of small dictionaries the four launches less count more than that (512 rows
// of 64: a step of 88 us takes 75).
constexpr int kSerialPartials = 64;  // up to so many partial sums are added up one after the other
__global__ void __launch_bounds__(256)
colsum_adam_kernel(const ColsumAdamParams p) {
  pdl_wait();
  __shared__ float s_sum[8][256];
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (p.loss_out != nullptr && blockIdx.x == 0 && blockIdx.y == 0) {
    float den = 0.0f;
    if (p.loss_weight != nullptr) {
      for (int i = threadIdx.x; i < p.loss_rows; i += 256) den += p.loss_weight[i];
      den = warp_sum(den);
      if (lane == 0) s_sum[0][warp] = den;
      __syncthreads();
      den = 0.0f;
      for (int i = 0; i < 8; ++i) den += s_sum[0][i];
      __syncthreads();
    }
    if (threadIdx.x == 0) {
      den = p.loss_weight != nullptr ? den * p.loss_den : p.loss_den;
      float sum = p.loss_sum[0];
      p.loss_sum[0] = 0.0f;
      if (p.loss_sum2 != nullptr) {
        const float sum2 = p.loss_sum2[0];
        p.loss_sum2[0] = 0.0f;
        if (p.loss_out2 != nullptr) p.loss_out2[0] = __fdiv_rn(sum2, den);
        sum += sum2;
      }
      p.loss_out[0] = __fdiv_rn(sum, den);
    }
  }
  if (p.n_seg == 0) return;
  int si = 0;
  while (si + 1 < p.n_seg && (int)blockIdx.x >= p.seg[si + 1].first_block) ++si;
  const ColsumAdamSeg g = p.seg[si];
  const int col0 = ((int)blockIdx.x - g.first_block) * 256;
  const int col = col0 + lane * 8;
  const int r0 = blockIdx.y * p.rows_per_block, r1 = min(p.rows, r0 + p.rows_per_block);
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
  if (col < g.d) {  // (d is a multiple of 8)
    for (int r = r0 + warp; r < r1; r += 32) {
      uint4 u[4];
#pragma unroll
      for (int q = 0; q < 4; ++q)
        u[q] = r + q * 8 < r1 ? __ldg(reinterpret_cast<const uint4*>(g.a + (size_t)(r + q * 8) * g.d + col)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float x[8];
        bf16x8_to_float(u[q], x);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += x[i];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) s_sum[warp][i * 32 + lane] = acc[i];  // column lane * 8 + i (no bank conflicts)
  __syncthreads();
  float s = 0.0f;
#pragma unroll
  for (int w = 0; w < 8; ++w) s += s_sum[w][threadIdx.x];
  const int c = col0 + (threadIdx.x & 31) * 8 + (threadIdx.x >> 5);
  if (gridDim.y > 1) {
    float* part = p.partial + (size_t)blockIdx.x * gridDim.y * 256;
    __stcg(part + blockIdx.y * 256 + threadIdx.x, s);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(p.counters + blockIdx.x, 1) == (int)gridDim.y - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (gridDim.y <= kSerialPartials) {
      s = 0.0f;
#pragma unroll 8
      for (int b = 0; b < (int)gridDim.y; ++b) s += __ldcg(part + b * 256 + threadIdx.x);
    } else {  // every warp an eighth of them, eight columns a lane
      float sum[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) sum[i] = 0.0f;
#pragma unroll 4
      for (int b = warp; b < (int)gridDim.y; b += 8) {
        const float4 u0 = __ldcg(reinterpret_cast<const float4*>(part + b * 256) + lane), u1 = __ldcg(reinterpret_cast<const float4*>(part + b * 256) + 32 + lane);
        sum[0] += u0.x; sum[1] += u0.y; sum[2] += u0.z; sum[3] += u0.w;
        sum[4] += u1.x; sum[5] += u1.y; sum[6] += u1.z; sum[7] += u1.w;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) s_sum[warp][(i >> 2) * 128 + lane * 4 + (i & 3)] = sum[i];
      __syncthreads();
      s = 0.0f;
#pragma unroll
      for (int w = 0; w < 8; ++w) s += s_sum[w][threadIdx.x];
    }
    if (threadIdx.x == 0) p.counters[blockIdx.x] = 0;  // for the next launch
  }
  if (c >= g.d || (p.status != nullptr && *reinterpret_cast<const volatile int*>(p.status) != 0)) return;  // see sparse_grad_adam_kernel
  float pi = g.p[c], mi = g.m[c], vi = g.v[c];
  adam_elem(pi, mi, vi, s, p.h);
  g.p[c] = pi; g.m[c] = mi; g.v[c] = vi;
}

// g [rows, d] keeps its values where mask [rows, d] (rows ld elements apart) is not zero and becomes zero elsewhere, in place, and the column
// sums of what is kept go to part [gridDim.y][d] (one row per block of rows; added up by the caller). Bound by memory: 4096 x 9216: 226 MB.
// As tensor operations (comparison, product, sum): 86 + 127 + 28 us; here 33.
__global__ void __launch_bounds__(256)
mask_colsum_kernel(__nv_bfloat16* __restrict__ g, const __nv_bfloat16* __restrict__ mask, long long ld, int rows, int d, int rows_per_block, float* __restrict__ part) {
  pdl_wait();
  __shared__ float s_sum[8][256];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int col0 = blockIdx.x * 256, col = col0 + lane * 8;
  const int r0 = blockIdx.y * rows_per_block, r1 = min(rows, r0 + rows_per_block);
  float acc[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
  if (col < d) {  // (d is a multiple of 8)
    for (int r = r0 + warp; r < r1; r += 32) {
      uint4 u[4], m[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (r + q * 8 < r1) {
          u[q] = *reinterpret_cast<const uint4*>(g + (size_t)(r + q * 8) * d + col);
          m[q] = __ldg(reinterpret_cast<const uint4*>(mask + (r + q * 8) * ld + col));
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (r + q * 8 >= r1) continue;
        uint32_t w[4] = {u[q].x, u[q].y, u[q].z, u[q].w};
        const uint32_t k[4] = {m[q].x, m[q].y, m[q].z, m[q].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if ((k[i] & 0x7fffu) == 0u) w[i] &= 0xffff0000u;
          if ((k[i] & 0x7fff0000u) == 0u) w[i] &= 0xffffu;
          acc[2 * i] += __uint_as_float(w[i] << 16);
          acc[2 * i + 1] += __uint_as_float(w[i] & 0xffff0000u);
        }
        *reinterpret_cast<uint4*>(g + (size_t)(r + q * 8) * d + col) = make_uint4(w[0], w[1], w[2], w[3]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) s_sum[warp][i * 32 + lane] = acc[i];
  __syncthreads();
  float s = 0.0f;
#pragma unroll
  for (int w = 0; w < 8; ++w) s += s_sum[w][threadIdx.x];
  const int c = col0 + (threadIdx.x & 31) * 8 + (threadIdx.x >> 5);
  if (c < d) part[(size_t)blockIdx.y * d + c] = s;
}

int mask_colsum_launch(__nv_bfloat16* g, const __nv_bfloat16* mask, long long ld, int rows, int d, int row_blocks, float* part, cudaStream_t stream) {
  if (d % 8 != 0 || ld % 8 != 0 || rows < 0 || row_blocks < 1) return (int)cudaErrorInvalidValue;
  if (d == 0) return 0;
  const int rpb = (rows + row_blocks - 1) / row_blocks;
  launch(mask_colsum_kernel, dim3((d + 255) / 256, row_blocks), 256, 0, stream, g, mask, ld, rows, d, rpb, part);
  return (int)cudaGetLastError();
}

// Row blocks for a launch of `col_blocks` blocks of 256 columns: eight CTAs per SM (2048 rows of 17152: 28 us with four, 22 with eight), at least
// 32 rows each, and no more than 64 partial sums to add up (4096 rows of 768: 9.6 us with 64, 11.0 with 128) while that leaves a block 64
// rows or less; with more rows a block of 64 to itself, up to 512 blocks, whose sums all warps add up (65536 rows of 64: 74 us with 64 blocks, 27 so;
// 262144 of 128: 258 and 45; 65536 of 768: 87 and 45).
int colsum_adam_row_blocks(int col_blocks, int rows) {
  int n = 1184 / (col_blocks > 0 ? col_blocks : 1);
  const int most = rows <= 64 * kSerialPartials ? (rows + 31) / 32 : (rows + 63) / 64, cap = rows <= 64 * kSerialPartials ? kSerialPartials : 512;
  n = n < most ? n : most;
  return n < 1 ? 1 : (n > cap ? cap : n);
}

int colsum_adam_launch(ColsumAdamParams p, int col_blocks, cudaStream_t stream) {
  if (p.n_seg < 0 || p.n_seg > kMaxColsumSegs || (p.n_seg > 0 && (p.rows <= 0 || col_blocks <= 0))) return (int)cudaErrorInvalidValue;
  if (p.n_seg == 0 && p.loss_out == nullptr) return 0;
  const int rb = p.n_seg > 0 ? colsum_adam_row_blocks(col_blocks, p.rows) : 1;
  p.rows_per_block = (p.rows + rb - 1) / rb;
  launch(colsum_adam_kernel, dim3(p.n_seg > 0 ? col_blocks : 1, rb), 256, 0, stream, p);
  return (int)cudaGetLastError();
}

// Flat Adam (torch.optim.Adam semantics without weight decay / amsgrad), optional bf16 shadow and
// squared-gradient accumulation. Used for small dense parameters (b_D, thresholds) and by the generic
// multi-tensor optimizer.
// VEC 4 reads and writes 16 bytes at a time (parameters, gradients and moments on 16-byte boundaries, the shadow on 8; what is left
// over of a length that is not a multiple of four goes element by element): 6.3 M parameters with shadow 32 us, 5.9 TB/s.
template <int VEC>
__global__ void __launch_bounds__(256)
adam_flat_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v,
                 long long n, AdamHyper h, const float* __restrict__ grad_mul, __nv_bfloat16* __restrict__ shadow,
                 float* __restrict__ grad_sq_sum, int update, const int* __restrict__ status) {
  pdl_wait();
  __shared__ float s_gsq[8];
  if (status != nullptr && *reinterpret_cast<const volatile int*>(status) != 0) return;  // see sparse_grad_adam_kernel
  const float gmul = grad_mul != nullptr ? *grad_mul : 1.0f;
  float gsq = 0.0f;
  const long long first = blockIdx.x * 256LL + threadIdx.x, stride = (long long)gridDim.x * 256;
  const long long n_vec = VEC == 4 ? n / 4 : 0;
  if constexpr (VEC == 4) {
    for (long long i = first; i < n_vec; i += stride) {
      float4 gi = reinterpret_cast<const float4*>(g)[i];
      gi.x *= gmul; gi.y *= gmul; gi.z *= gmul; gi.w *= gmul;
      gsq += gi.x * gi.x + gi.y * gi.y + gi.z * gi.z + gi.w * gi.w;
      if (update) {
        float4 pi = reinterpret_cast<float4*>(p)[i], mi = reinterpret_cast<float4*>(m)[i], vi = reinterpret_cast<float4*>(v)[i];
        adam_elem(pi.x, mi.x, vi.x, gi.x, h); adam_elem(pi.y, mi.y, vi.y, gi.y, h);
        adam_elem(pi.z, mi.z, vi.z, gi.z, h); adam_elem(pi.w, mi.w, vi.w, gi.w, h);
        reinterpret_cast<float4*>(p)[i] = pi;
        reinterpret_cast<float4*>(m)[i] = mi;
        reinterpret_cast<float4*>(v)[i] = vi;
        if (shadow != nullptr) reinterpret_cast<uint2*>(shadow)[i] = make_uint2(pack_bf16x2(pi.x, pi.y), pack_bf16x2(pi.z, pi.w));
      }
    }
  }
  for (long long i = n_vec * 4 + first; i < n; i += stride) {
    const float gi = g[i] * gmul;
    gsq += gi * gi;
    if (update) {
      float pi = p[i], mi = m[i], vi = v[i];
      adam_elem(pi, mi, vi, gi, h);
      p[i] = pi; m[i] = mi; v[i] = vi;
      if (shadow != nullptr) shadow[i] = __float2bfloat16(pi);
    }
  }
  if (grad_sq_sum != nullptr) {
    gsq = warp_sum(gsq);
    if ((threadIdx.x & 31) == 0) s_gsq[threadIdx.x >> 5] = gsq;
    __syncthreads();
    if (threadIdx.x < 32) {
      float t = threadIdx.x < 8 ? s_gsq[threadIdx.x] : 0.0f;
      t = warp_sum(t);
      if (threadIdx.x == 0) atomicAdd(grad_sq_sum, t);
    }
  }
}

int adam_flat_launch(float* p, const float* g, float* m, float* v, long long n, AdamHyper h, const float* grad_mul,
                     __nv_bfloat16* shadow, float* grad_sq_sum, int update, const int* status, cudaStream_t stream) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(p) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(m) | reinterpret_cast<uintptr_t>(v);
  const bool wide = at % 16 == 0 && reinterpret_cast<uintptr_t>(shadow) % 8 == 0 && n >= 4096;  // (short ones: more threads instead)
  long long blocks = ((wide ? n / 4 : n) + 255) / 256;
  if (blocks > 148 * 16) blocks = 148 * 16;
  if (blocks < 1) blocks = 1;
  auto kern = wide ? adam_flat_kernel<4> : adam_flat_kernel<1>;
  launch(kern, (int)blocks, 256, 0, stream, p, g, m, v, n, h, grad_mul, shadow, grad_sq_sum, update, status);
  return (int)cudaGetLastError();
}

// Row L2 norms of an fp32 [F, d] matrix (+ optional bf16 shadow refresh): used at set-up and after
// loading weights so that dec_norm / shadows agree with the master copy.
__global__ void __launch_bounds__(256)
row_norm_shadow_kernel(const float* __restrict__ W, int F, int d, float* __restrict__ norm,
                       __nv_bfloat16* __restrict__ shadow) {
  __shared__ float s_red[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int f = blockIdx.x; f < F; f += gridDim.x) {
    float s = 0.0f;
    for (int c = threadIdx.x; c < d; c += 256) {
      const float w = W[(size_t)f * d + c];
      s = fmaf(w, w, s);
      if (shadow != nullptr) shadow[(size_t)f * d + c] = __float2bfloat16(w);
    }
    s = warp_sum(s);
    __syncthreads();
    if (lane == 0) s_red[warp] = s;
    __syncthreads();
    if (warp == 0) {
      float t = lane < 8 ? s_red[lane] : 0.0f;
      t = warp_sum(t);
      if (lane == 0 && norm != nullptr) norm[f] = sqrtf(t);
    }
  }
}

int row_norm_shadow_launch(const float* W, int F, int d, float* norm, __nv_bfloat16* shadow, cudaStream_t stream) {
  int blocks = F < 148 * 16 ? F : 148 * 16;
  launch_plain(row_norm_shadow_kernel, blocks, 256, 0, stream, W, F, d, norm, shadow);
  return (int)cudaGetLastError();
}

}  // namespace lmsae
