// mlp_kernels.cu -- element-wise and reduction kernels of the learned-entry
// MLP (BF16 storage, FP32 arithmetic).  The GEMMs are gemm_tc.cu.
#include <algorithm>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mlp_kernels.h"

namespace rte {

// out[r][c] = bf16(x[r][c] * scale) for c < d, 0 for d <= c < dp.
__global__ void cast_rows_bf16_k(const float* __restrict__ x, int64_t rows, int d, int ld,
                                 float scale, int dp, __nv_bfloat16* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * dp) return;
  const int64_t r = i / dp;
  const int c = (int)(i % dp);
  out[i] = __float2bfloat16_rn(c < d ? x[r * ld + c] * scale : 0.0f);
}

// out[c][r] = in[r][c] through 64x64 shared-memory tiles: 16-byte loads and
// stores, four lanes to a 64-byte run of an output row.  C is a multiple of 8
// and `in` 16-byte aligned; output rows of R % 8 != 0 elements are stored one
// by one.  Tile rows are 33 words apart, which keeps both the row-wise stores
// and the column-wise reads off each other's banks.  On one GB300 the step's
// eight transposes (4096 x 4096 and smaller) took 71 us through 32x32 tiles
// of 2-byte accesses, now 37 us.
constexpr int kTrTile = 64;
__global__ void __launch_bounds__(256) transpose_bf16_k(const uint16_t* __restrict__ in, int R, int C,
                                                        uint16_t* __restrict__ out) {
  __shared__ uint32_t t[kTrTile][kTrTile / 2 + 1];
  const int c0 = blockIdx.x * kTrTile, r0 = blockIdx.y * kTrTile;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int id = threadIdx.x + 256 * i;
    const int r = id >> 3, v = id & 7;
    if (r0 + r < R && c0 + 8 * v < C) {
      const uint4 x = *reinterpret_cast<const uint4*>(in + (int64_t)(r0 + r) * C + c0 + 8 * v);
      t[r][4 * v] = x.x;
      t[r][4 * v + 1] = x.y;
      t[r][4 * v + 2] = x.z;
      t[r][4 * v + 3] = x.w;
    }
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int id = threadIdx.x + 256 * i;
    // lanes: 4 groups of 8 rows, then 8 columns; warps: the other half of the rows, then 8 columns further
    const int c = ((id >> 2) & 7) | ((id >> 6) << 3), r = 8 * ((id & 3) | (((id >> 5) & 1) << 2));
    if (c0 + c >= C || r0 + r >= R) continue;
    uint32_t h[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) h[j] = (c & 1) ? t[r + j][c >> 1] >> 16 : t[r + j][c >> 1] & 0xffffu;
    uint16_t* o = out + (int64_t)(c0 + c) * R + r0 + r;
    if ((R & 7) == 0) {
      *reinterpret_cast<uint4*>(o) = make_uint4(h[0] | h[1] << 16, h[2] | h[3] << 16, h[4] | h[5] << 16, h[6] | h[7] << 16);
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (r0 + r + j < R) o[j] = (uint16_t)h[j];
    }
  }
}

// Row-wise softmax cross-entropy: loss[m] = logsumexp(z_m) - z_m[y_m];
// dz[m][c] = (softmax(z_m)[c] - [c == y_m]) * inv_m, stored as BF16.
// Thread t of the row's block takes columns t, t + 512, ...: with V > 0 (C up
// to 512 V) it keeps them in registers, so the row is read once and each
// exponential computed once; V = 0 reads them for each pass.  Both add in the
// same order.  At 4096 x 4096 on one GB300: 49 us in three passes, 25 us
// in one.
constexpr int kSoftmaxThreads = 512;
template <int V>
__global__ void __launch_bounds__(kSoftmaxThreads) softmax_ce_k(const float* __restrict__ z, int M, int C,
                                                                const int32_t* __restrict__ y, float inv_m,
                                                                __nv_bfloat16* __restrict__ dz,
                                                                float* __restrict__ loss) {
  const int m = blockIdx.x;
  const float* row = z + (int64_t)m * C;
  __shared__ float red[32];
  float v[V > 0 ? V : 1];
  float mx = -3.402823466e38f;
  if constexpr (V > 0) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int c = threadIdx.x + kSoftmaxThreads * k;
      v[k] = c < C ? row[c] : -3.402823466e38f;
    }
#pragma unroll
    for (int k = 0; k < V; ++k) mx = fmaxf(mx, v[k]);
  } else {
    for (int c = threadIdx.x; c < C; c += kSoftmaxThreads) mx = fmaxf(mx, row[c]);
  }
  for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
  if (threadIdx.x < 32) {
    float u = threadIdx.x < kSoftmaxThreads / 32 ? red[threadIdx.x] : -3.402823466e38f;
    for (int o = 16; o; o >>= 1) u = fmaxf(u, __shfl_xor_sync(0xffffffffu, u, o));
    if (threadIdx.x == 0) red[0] = u;
  }
  __syncthreads();
  mx = red[0];
  __syncthreads();
  float s = 0.f;
  if constexpr (V > 0) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int c = threadIdx.x + kSoftmaxThreads * k;
      if (c < C) {
        v[k] = __expf(v[k] - mx);
        s += v[k];
      }
    }
  } else {
    for (int c = threadIdx.x; c < C; c += kSoftmaxThreads) s += __expf(row[c] - mx);
  }
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    float u = threadIdx.x < kSoftmaxThreads / 32 ? red[threadIdx.x] : 0.f;
    for (int o = 16; o; o >>= 1) u += __shfl_xor_sync(0xffffffffu, u, o);
    if (threadIdx.x == 0) red[0] = u;
  }
  __syncthreads();
  const float sum = red[0];
  const float inv = 1.0f / sum;
  const int label = y[m];
  auto grad = [&](int c, float e) {
    float p = e * inv;
    if (c == label) p -= 1.0f;
    dz[(int64_t)m * C + c] = __float2bfloat16_rn(p * inv_m);
  };
  if constexpr (V > 0) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const int c = threadIdx.x + kSoftmaxThreads * k;
      if (c < C) grad(c, v[k]);
    }
  } else {
    for (int c = threadIdx.x; c < C; c += kSoftmaxThreads) grad(c, __expf(row[c] - mx));
  }
  if (threadIdx.x == 0 && loss) loss[m] = logf(sum) + mx - row[label];
}

// out = bf16(g * (h > 0)), four elements a thread (n is a multiple of 4).
__global__ void relu_grad_k(const float4* __restrict__ g, const uint2* __restrict__ h, int64_t n4,
                            uint2* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n4) return;
  const float4 a = g[i];
  const uint2 b = h[i];
  auto live = [](uint32_t bits) { return __uint_as_float(bits << 16) > 0.f; };
  const __nv_bfloat162 lo = __floats2bfloat162_rn(live(b.x & 0xffffu) ? a.x : 0.f, live(b.x >> 16) ? a.y : 0.f);
  const __nv_bfloat162 hi = __floats2bfloat162_rn(live(b.y & 0xffffu) ? a.z : 0.f, live(b.y >> 16) ? a.w : 0.f);
  out[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
}

// Column sums out[n] = sum over m of x[m][n] (BF16 input, FP32 sums) in two
// passes with a fixed order, so results are reproducible: block (bx, by)
// takes columns 64 bx .. 64 bx + 63 (two per thread; N is even) and row slice
// by (rows by*rs .. by*rs + rs - 1); its thread (c, r) sums rows r, r + 8,
// ... of the slice for columns 2c and 2c + 1, the eight row lanes are added in
// lane order, and part[by][n] receives the slice's sum.  The second pass adds
// the slices in order.
constexpr int kColSumRowLanes = 8;
__global__ void col_sum_part_k(const __nv_bfloat16* __restrict__ x, int M, int N, int rs,
                               float* __restrict__ part) {
  __shared__ float2 sh[kColSumRowLanes][32];
  const int c = threadIdx.x, r = threadIdx.y;
  const int n = 2 * (blockIdx.x * 32 + c);
  const int m0 = blockIdx.y * rs, m1 = min(M, m0 + rs);
  float2 s = make_float2(0.f, 0.f);
  if (n < N) {
#pragma unroll 8
    for (int m = m0 + r; m < m1; m += kColSumRowLanes) {
      const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(x + (int64_t)m * N + n);
      s.x += __bfloat162float(v.x);
      s.y += __bfloat162float(v.y);
    }
  }
  sh[r][c] = s;
  __syncthreads();
  if (r == 0 && n < N) {
    float2 t = sh[0][c];
#pragma unroll
    for (int i = 1; i < kColSumRowLanes; ++i) {
      t.x += sh[i][c].x;
      t.y += sh[i][c].y;
    }
    *reinterpret_cast<float2*>(part + (int64_t)blockIdx.y * N + n) = t;
  }
}

__global__ void col_sum_finish_k(const float* __restrict__ part, int slices, int N, float* __restrict__ out) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= N) return;
  float s = 0.f;
  for (int i = 0; i < slices; ++i) s += part[(int64_t)i * N + n];
  out[n] = s;
}

// Adam on FP32 master weights; refreshes the BF16 copies.  Every parameter
// tensor in one launch: tensor t owns blocks first[t] .. first[t + 1] - 1.
__global__ void adam_k(AdamArgs a) {
  int t = 0;
  while (t + 1 < kAdamTensors && (int)blockIdx.x >= a.t[t + 1].first) ++t;
  const AdamTensor& p = a.t[t];
  const int64_t i = (int64_t)(blockIdx.x - p.first) * blockDim.x + threadIdx.x;
  if (i >= p.n) return;
  const float gi = p.g[i];
  const float m = a.b1 * p.m1[i] + (1.f - a.b1) * gi;
  const float v = a.b2 * p.m2[i] + (1.f - a.b2) * gi * gi;
  p.m1[i] = m;
  p.m2[i] = v;
  const float upd = a.lr * (m * a.c1) / (sqrtf(v * a.c2) + a.eps);
  const float nw = p.w[i] - upd;
  p.w[i] = nw;
  if (p.w16) reinterpret_cast<__nv_bfloat16*>(p.w16)[i] = __float2bfloat16_rn(nw);
}

// Class of each base point: that of its kd-tree leaf (class_of_leaf[0] for a
// point that no leaf lists), then the class of each query's best point.
__global__ void fill_i32_k(int32_t* __restrict__ out, int64_t n, const int32_t* __restrict__ value) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = *value;
}
__global__ void point_class_k(const int32_t* __restrict__ pids, int64_t n, int cap, int64_t np,
                              const int32_t* __restrict__ class_of_leaf, int32_t* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t p = pids[i];
  if (p < np) out[p] = class_of_leaf[i / cap];
}
__global__ void label_k(const int32_t* __restrict__ ids, int64_t n, int64_t np,
                        const int32_t* __restrict__ point_class, const int32_t* __restrict__ class_of_leaf,
                        int32_t* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t p = ids[i];
  out[i] = p >= 0 && p < np ? point_class[p] : class_of_leaf[0];
}

__global__ void f32_to_bf16_k(const float* __restrict__ x, int64_t n, __nv_bfloat16* __restrict__ out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = __float2bfloat16_rn(x[i]);
}

// Rows of dp BF16 values (a multiple of 8) in 16-byte pieces.
__global__ void gather_rows_k(const uint4* __restrict__ src, int pieces, const int64_t* __restrict__ idx, int rows,
                              const int32_t* __restrict__ labels_src, uint4* __restrict__ dst,
                              int32_t* __restrict__ labels_dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= rows * pieces) return;
  const int r = i / pieces, c = i - r * pieces;
  const int64_t s = idx[r];
  dst[i] = src[s * pieces + c];
  if (c == 0) labels_dst[r] = labels_src[s];
}

// argmax key -> class column; class -> leaf through class_leaf (null: identity).
// A zero key (no column was a maximum: every logit NaN) gives -1.
__global__ void argmax_to_leaf_k(const unsigned long long* __restrict__ keys, int n,
                                 const int32_t* __restrict__ class_leaf, int32_t* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (keys[i] == 0ull) {
    out[i] = -1;
    return;
  }
  const int col = 0x7fffffff - (int)(keys[i] & 0xffffffffu);
  out[i] = class_leaf ? class_leaf[col] : col;
}

static unsigned blocks(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

cudaError_t launch_cast_rows_bf16(const float* x, int64_t rows, int d, int ld, float scale, int dp,
                                  void* out, cudaStream_t st) {
  if (rows == 0) return cudaSuccess;
  cast_rows_bf16_k<<<blocks(rows * dp, 256), 256, 0, st>>>(x, rows, d, ld, scale, dp,
                                                          (__nv_bfloat16*)out);
  return cudaGetLastError();
}
cudaError_t launch_transpose_bf16(const void* in, int R, int C, void* out, cudaStream_t st) {
  if (C & 7) return cudaErrorInvalidValue;
  dim3 grid((C + kTrTile - 1) / kTrTile, (R + kTrTile - 1) / kTrTile);
  transpose_bf16_k<<<grid, 256, 0, st>>>((const uint16_t*)in, R, C, (uint16_t*)out);
  return cudaGetLastError();
}
cudaError_t launch_softmax_ce(const float* z, int M, int C, const int32_t* y, float inv_m, void* dz,
                              float* loss, cudaStream_t st) {
  __nv_bfloat16* d = (__nv_bfloat16*)dz;
  if (C <= 4 * kSoftmaxThreads)
    softmax_ce_k<4><<<M, kSoftmaxThreads, 0, st>>>(z, M, C, y, inv_m, d, loss);
  else if (C <= 8 * kSoftmaxThreads)
    softmax_ce_k<8><<<M, kSoftmaxThreads, 0, st>>>(z, M, C, y, inv_m, d, loss);
  else if (C <= 16 * kSoftmaxThreads)
    softmax_ce_k<16><<<M, kSoftmaxThreads, 0, st>>>(z, M, C, y, inv_m, d, loss);
  else
    softmax_ce_k<0><<<M, kSoftmaxThreads, 0, st>>>(z, M, C, y, inv_m, d, loss);
  return cudaGetLastError();
}
cudaError_t launch_relu_grad(const float* g, const void* h, int64_t n, void* out, cudaStream_t st) {
  if (n & 3) return cudaErrorInvalidValue;
  relu_grad_k<<<blocks(n / 4, 256), 256, 0, st>>>((const float4*)g, (const uint2*)h, n / 4, (uint2*)out);
  return cudaGetLastError();
}
int col_sum_slices(int M) { return std::max(1, std::min(kColSumMaxSlices, M / 256)); }
cudaError_t launch_col_sum_bf16(const void* x, int M, int N, float* out, float* part, cudaStream_t st) {
  const int slices = col_sum_slices(M);
  const int rs = (M + slices - 1) / slices;
  if (N & 1) return cudaErrorInvalidValue;
  col_sum_part_k<<<dim3((N + 63) / 64, slices), dim3(32, kColSumRowLanes), 0, st>>>(
      (const __nv_bfloat16*)x, M, N, rs, part);
  col_sum_finish_k<<<blocks(N, 256), 256, 0, st>>>(part, slices, N, out);
  return cudaGetLastError();
}
cudaError_t launch_adam(AdamArgs a, cudaStream_t st) {
  int first = 0;
  for (int t = 0; t < kAdamTensors; ++t) {
    a.t[t].first = first;
    first += (int)blocks(a.t[t].n, 256);
  }
  adam_k<<<first, 256, 0, st>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_point_labels(const int32_t* ids, int64_t n, const int32_t* pids, int64_t n_leaves, int cap,
                                int64_t np, const int32_t* class_of_leaf, int32_t* point_class, int32_t* labels,
                                cudaStream_t st) {
  fill_i32_k<<<blocks(np, 256), 256, 0, st>>>(point_class, np, class_of_leaf);
  point_class_k<<<blocks(n_leaves * cap, 256), 256, 0, st>>>(pids, n_leaves * cap, cap, np, class_of_leaf,
                                                             point_class);
  label_k<<<blocks(n, 256), 256, 0, st>>>(ids, n, np, point_class, class_of_leaf, labels);
  return cudaGetLastError();
}
cudaError_t launch_f32_to_bf16(const float* x, int64_t n, void* out, cudaStream_t st) {
  f32_to_bf16_k<<<blocks(n, 256), 256, 0, st>>>(x, n, (__nv_bfloat16*)out);
  return cudaGetLastError();
}
cudaError_t launch_gather_rows(const void* src, int dp, const int64_t* idx, int rows,
                               const int32_t* labels_src, void* dst, int32_t* labels_dst,
                               cudaStream_t st) {
  if (dp & 7) return cudaErrorInvalidValue;
  gather_rows_k<<<blocks((int64_t)rows * (dp / 8), 256), 256, 0, st>>>(
      (const uint4*)src, dp / 8, idx, rows, labels_src, (uint4*)dst, labels_dst);
  return cudaGetLastError();
}
cudaError_t launch_argmax_to_leaf(const unsigned long long* keys, int n, const int32_t* class_leaf,
                                  int32_t* out, cudaStream_t st) {
  if (n == 0) return cudaSuccess;
  argmax_to_leaf_k<<<blocks(n, 256), 256, 0, st>>>(keys, n, class_leaf, out);
  return cudaGetLastError();
}

}  // namespace rte
