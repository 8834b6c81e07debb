// knn_graph.cu -- exact k-nearest-neighbour graph of a base, on the GPU.
//
// The reference loads its proximity graph from a file and has no builder
// (graph.cu:120).  This builds the degree-R exact kNN graph that its search
// runs on: row i lists the R nearest rows j != i by exact squared L2
// distance (FP64), in (distance, id) order.
//
//   0. The rows are centred on their column mean mu (FP64 sums in a fixed
//      order, rounded to FP32): c = fl(x - mu).  Distances do not change
//      under a shift, and the error bound of step 3 scales with the norms of
//      what the GEMM multiplies, so centring tightens it by |x| / |c| (about
//      5x for values in [0, 1] around 0.5).
//   1. Each centred row c is split into BF16 c_hi = bf16(c) and
//      c_lo = bf16(c - c_hi);
//      A = [hi | hi | lo] and B = [hi | lo | hi] along K, so one tensor-core
//      GEMM (gemm_tc.cu, K = 3*dp) gives hi.hi + hi.lo + lo.hi, the dot
//      product to about 2^-16 relative.
//   2. Block of rows by block of rows: a threshold per row from a sample of
//      the columns (sample_threshold), then one tensor-core pass over all
//      columns that keeps those whose approximate distance
//      |x|^2 + |y|^2 - 2 x.y lies below it (knn_filter.cu): a few hundred per
//      row, with no n^2 array in memory.
//   3. finish_rows: with a_R the R-th smallest approximate distance and err
//      the approximation's error bound, every true neighbour has an
//      approximate distance of at most a_R + 2 err.  If that is below the
//      threshold (so all such columns were kept), those few get exact FP64
//      distances and are sorted by (distance, id): the row is exact.
//   4. Rows that step 3 cannot certify (more such columns than it holds, a
//      threshold that came out too small or a list that overflowed), and
//      every row of a small base or of a degree above 128: the dot products
//      of a block of such rows in memory, the K = 2R + 32 smallest per row
//      (select_rows) and a lower bound on every column left out, exact FP64
//      distances (rerank_rows).  The row is certified exact when its R-th
//      distance is below the left-out bound minus err; rows that fail are
//      redone with 1024 candidates from the same block of dot products, and a
//      row that fails again is an error.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cmath>
#include <vector>

#include "gemm_tc.h"
#include "knn_filter.h"
#include "index_impl.h"
#include "rtentry.h"
#include "widen.cuh"

namespace rte {
namespace {

constexpr int kSelThreads = 256;
constexpr int kSelT = 16;                         // candidates kept per thread
constexpr int kSelPool = kSelThreads * kSelT;     // 4096 merged per row
constexpr int kMaxCand = 1024;                    // the retry's candidate count

// The thresholded pass serves degrees of up to 128 and bases of at least 1024
// rows; below, the dot products in memory take less.
constexpr int kFilterMaxDegree = 128;
constexpr int64_t kFilterMinRows = 1024;
constexpr int kFinRows = 8;  // rows per block of finish_rows

// Sizes of the thresholded pass.
struct FilterPlan {
  bool use;        // false: stored products for every row
  int64_t sample;  // columns sampled for the thresholds
  int rank;        // a row's threshold: its rank-th smallest sampled distance
  int cap;         // list slots per row
  int kmax;        // candidates per row that finish_rows measures
  int64_t block;   // rows per launch
};

constexpr int kMaxCap = 4096;     // list slots per row at most
constexpr int kMaxFinish = 512;   // candidates per row that finish_rows measures at most
size_t finish_smem(int cap, int kmax) { return (size_t)kFinRows * (12 * (size_t)kmax + 4 * (size_t)cap); }

FilterPlan filter_plan(int64_t n, int degree) {
  FilterPlan p{};
  if (degree > kFilterMaxDegree || n < kFilterMinRows) return p;
  // About `want` columns are kept per row: enough that the R-th smallest plus
  // twice the error bound lies well below the threshold.  The sample is a 24th
  // of the base, so the threshold is about its 10th smallest distance at degree
  // 32, and the kept count spreads by a third.  It keeps growing with the base
  // (up to 524,288 columns, whose block of dot products takes 8.6 GB): held at
  // 65,536, 628,083 of 5M x 32 rows' lists overflowed and their dot products
  // were stored, 27.4 s in all, now none and 18.2 s.
  const int64_t want = 4 * (int64_t)degree + 96;
  p.sample = std::min<int64_t>(std::max<int64_t>(n / 24, 256), 524288);
  p.rank = (int)std::max<int64_t>(8, (want * p.sample + n - 1) / n) + 1;  // the row itself may be sampled
  p.kmax = 64;
  while (p.kmax < 2 * degree + 32) p.kmax <<= 1;  // kMaxFinish at degree 128
  // The count of columns below the rank-th smallest of the sample has mean
  // rank n / sample and a relative spread of 1 / sqrt(rank): a list holds four
  // spreads more, and the slots reserved and not used.
  const double kept = (double)n / (double)p.sample * (p.rank + 4.0 * std::sqrt((double)p.rank) + 4.0) + 128.0;
  p.cap = degree <= 64 ? 1024 : 2048;
  while (p.cap < kept && p.cap < kMaxCap) p.cap <<= 1;  // 180 KB of shared memory at degree 128
  p.use = p.cap >= kept;  // past about 90M rows most lists would overflow
  // rows per launch: dot products with the sample of up to 1 GB, and of 4096
  // rows at least (the pass reads the whole base for each block)
  p.block = std::min<int64_t>(16384, std::max<int64_t>(4096, ((1ll << 30) / (p.sample * 4)) / 128 * 128));
  p.block = std::min<int64_t>(p.block, n);
  return p;
}

constexpr int kMeanSlices = 256;  // row slices of the column mean's first pass

// Column sums of row slice blockIdx.y in FP64 (rows in order), one thread
// per column: part[slice][c].
__global__ void col_sum_slices(const float* __restrict__ x, int64_t n, int d, double* __restrict__ part) {
  const int s = blockIdx.y;
  const int64_t r0 = n * s / kMeanSlices, r1 = n * (s + 1) / kMeanSlices;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < d; c += gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int64_t r = r0; r < r1; ++r) acc += (double)__ldg(x + r * d + c);
    part[(int64_t)s * d + c] = acc;
  }
}

// mu[c] = (sum of the slices' sums in slice order) / n, rounded to FP32.
__global__ void col_mean_finish(const double* __restrict__ part, int64_t n, int d, float* __restrict__ mu) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= d) return;
  double acc = 0.0;
  for (int s = 0; s < kMeanSlices; ++s) acc += part[(int64_t)s * d + c];
  mu[c] = (float)(acc / (double)n);
}

// Centring, split and norms of the centred rows: one warp per row.
__global__ void split_rows(const float* __restrict__ x, const float* __restrict__ mu, int64_t n, int d,
                           int dp, __nv_bfloat16* __restrict__ a, __nv_bfloat16* __restrict__ b,
                           float* __restrict__ nrm32, double* __restrict__ nrm64,
                           unsigned long long* __restrict__ max_nrm) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t ld = 3 * (int64_t)dp;
  double top = 0.0;  // the largest squared norm (non-negative doubles order as their bits)
  for (int64_t r = warp; r < n; r += nwarps) {
    double s = 0.0;
    for (int c = lane; c < dp; c += 32) {
      const float v = c < d ? __fsub_rn(x[r * d + c], mu[c]) : 0.0f;
      const __nv_bfloat16 hi = __float2bfloat16_rn(v);
      const __nv_bfloat16 lo = __float2bfloat16_rn(__fsub_rn(v, __bfloat162float(hi)));
      a[r * ld + c] = hi;           // A = [hi | hi | lo]
      a[r * ld + dp + c] = hi;
      a[r * ld + 2 * dp + c] = lo;
      b[r * ld + c] = hi;           // B = [hi | lo | hi]
      b[r * ld + dp + c] = lo;
      b[r * ld + 2 * dp + c] = hi;
      s += (double)v * (double)v;
    }
    for (int off = 16; off >= 1; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (lane == 0) {
      nrm64[r] = s;
      nrm32[r] = (float)s;
      top = fmax(top, s);
    }
  }
  if (lane == 0 && top > 0.0) atomicMax(max_nrm, (unsigned long long)__double_as_longlong(top));
}

// |approximate - exact| <= err for every column: the hi/lo split and the
// FP32 sums over the centred rows (norms qnorm, at most max_norm), plus the
// centring's rounding -- each fl(x - mu) is off by at most 2^-24 of |x - mu|,
// which moves a squared distance by at most about 2^-23 (qnorm + max_norm)^2;
// the last term doubles that for room.
__device__ __forceinline__ double approx_error(double nrm, double max_norm, int d) {
  const double qnorm = sqrt(nrm);
  return (ldexp(1.0, -14) + d * ldexp(1.0, -21)) * qnorm * max_norm +
         ldexp(1.0, -20) * (nrm + max_norm * max_norm) +
         ldexp(1.0, -22) * (qnorm + max_norm) * (qnorm + max_norm);
}

__device__ __forceinline__ bool key_less(float da, int ia, float db, int ib) {
  return da < db || (da == db && ia < ib);
}

// In-place ascending bitonic sort of kSelPool (distance, id) pairs in shared
// memory by all threads of the block.
__device__ void block_sort(float* sd, int* si) {
  for (int step = 2; step <= kSelPool; step <<= 1)
    for (int sub = step >> 1; sub >= 1; sub >>= 1) {
      for (int i = threadIdx.x; i < kSelPool; i += blockDim.x) {
        const int j = i ^ sub;
        if (j > i) {
          const bool up = (i & step) == 0;
          const bool sw = up ? key_less(sd[j], si[j], sd[i], si[i]) : key_less(sd[i], si[i], sd[j], si[j]);
          if (sw) {
            const float t = sd[i];
            sd[i] = sd[j];
            sd[j] = t;
            const int u = si[i];
            si[i] = si[j];
            si[j] = u;
          }
        }
      }
      __syncthreads();
    }
}

// One block per row: approximate distances from the dot products in
// D[row][0..n), the K smallest by (distance, id), and the smallest
// approximate distance any left-out column can have.
// Row r of the block of dot products is row rows[r] of the base; with
// `local`, block i serves row local[i] of it.
__global__ void __launch_bounds__(kSelThreads) select_rows(const float* __restrict__ D, int64_t ld,
                                                           const int64_t* __restrict__ rows, int64_t n,
                                                           const float* __restrict__ nrm32, int K,
                                                           const int32_t* __restrict__ local,
                                                           int32_t* __restrict__ cand,
                                                           float* __restrict__ excl) {
  __shared__ float sd[kSelPool];
  __shared__ int si[kSelPool];
  __shared__ float sdrop[kSelThreads];
  const int r = local ? local[blockIdx.x] : (int)blockIdx.x;
  const float qn = nrm32[rows[r]];
  float kd[kSelT];
  int ki[kSelT];
#pragma unroll
  for (int s = 0; s < kSelT; ++s) {
    kd[s] = INFINITY;
    ki[s] = INT32_MAX;
  }
  const float* row = D + (int64_t)r * ld;
  // Eight columns' loads are in flight ahead of the insertions, in code: left to
  // the compiler the loop took 76 ms in one form and 90 ms in another that only
  // loads qn differently (100k x 64, degree 129: the whole build 134 and 147 ms,
  // 132 ms now; four columns ahead 161 ms).
  constexpr int kAhead = 8;
  for (int64_t j0 = threadIdx.x; j0 < n; j0 += kSelThreads * kAhead) {
    float a[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int64_t j = j0 + kSelThreads * u;
      a[u] = j < n ? __fmaf_rn(-2.0f, __ldg(row + j), __fadd_rn(qn, __ldg(nrm32 + j))) : INFINITY;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (a[u] < kd[kSelT - 1]) {  // insert, keeping the list sorted (ties keep scan order)
        float cd = a[u];
        int ci = (int)(j0 + kSelThreads * u);
#pragma unroll
        for (int s = 0; s < kSelT; ++s)
          if (cd < kd[s]) {
            const float t = kd[s];
            kd[s] = cd;
            cd = t;
            const int v = ki[s];
            ki[s] = ci;
            ci = v;
          }
      }
    }
  }
  // what this thread dropped is no smaller than its last kept value (when full)
  sdrop[threadIdx.x] = ki[kSelT - 1] != INT32_MAX ? kd[kSelT - 1] : INFINITY;
#pragma unroll
  for (int s = 0; s < kSelT; ++s) {
    sd[threadIdx.x * kSelT + s] = kd[s];
    si[threadIdx.x * kSelT + s] = ki[s];
  }
  __syncthreads();
  block_sort(sd, si);
  const int64_t o = blockIdx.x;
  for (int k = threadIdx.x; k < K; k += kSelThreads) cand[o * K + k] = si[k] < n ? si[k] : -1;
  if (threadIdx.x == 0) {
    float m = K < kSelPool ? sd[K] : INFINITY;
    for (int t = 0; t < kSelThreads; ++t) m = fminf(m, sdrop[t]);
    excl[o] = m;
  }
}

__device__ __forceinline__ bool key_less64(double da, int ia, double db, int ib) {
  return da < db || (da == db && ia < ib);
}

// One block per row: exact FP64 distances of the candidates, sorted by
// (distance, id) with the row itself excluded; certified when the R-th
// distance is below the left-out bound minus the error bound.
__global__ void __launch_bounds__(256) rerank_rows(const float* __restrict__ x, int d, const int64_t* __restrict__ rows,
                                                   const int32_t* __restrict__ cand, int K, int Kp,
                                                   const float* __restrict__ excl,
                                                   const double* __restrict__ nrm64,
                                                   const unsigned long long* __restrict__ max_nrm,
                                                   int R, int32_t* __restrict__ out,
                                                   int* __restrict__ failed) {
  extern __shared__ unsigned char sm_raw[];
  double* sd = reinterpret_cast<double*>(sm_raw);
  int* si = reinterpret_cast<int*>(sd + Kp);
  const int r = blockIdx.x;
  const int64_t gi = rows[r];
  const float* q = x + gi * d;
  for (int k = threadIdx.x; k < Kp; k += blockDim.x) {
    const int id = k < K ? cand[(int64_t)r * K + k] : -1;
    double s = INFINITY;
    if (id >= 0 && id != gi) {
      const float* p = x + (int64_t)id * d;
      s = 0.0;
      for (int c = 0; c < d; ++c) {
        const double t = (double)__ldg(p + c) - (double)__ldg(q + c);
        s = fma(t, t, s);
      }
    }
    sd[k] = s;
    si[k] = id >= 0 && id != gi ? id : INT32_MAX;
  }
  __syncthreads();
  for (int step = 2; step <= Kp; step <<= 1)
    for (int sub = step >> 1; sub >= 1; sub >>= 1) {
      for (int i = threadIdx.x; i < Kp; i += blockDim.x) {
        const int j = i ^ sub;
        if (j > i) {
          const bool up = (i & step) == 0;
          const bool sw = up ? key_less64(sd[j], si[j], sd[i], si[i]) : key_less64(sd[i], si[i], sd[j], si[j]);
          if (sw) {
            const double t = sd[i];
            sd[i] = sd[j];
            sd[j] = t;
            const int u = si[i];
            si[i] = si[j];
            si[j] = u;
          }
        }
      }
      __syncthreads();
    }
  const double err = approx_error(nrm64[gi], sqrt(__longlong_as_double((long long)*max_nrm)), d);
  if (threadIdx.x == 0) {
    const bool ok = si[R - 1] != INT32_MAX && sd[R - 1] < (double)excl[r] - err;
    if (!ok) atomicAdd(failed, 1);
    out[gi * R] = ok ? si[0] : -1;  // -1 marks the row for the retry
  }
  __syncthreads();
  if (out[gi * R] >= 0)
    for (int k = threadIdx.x + 1; k < R; k += blockDim.x) out[gi * R + k] = si[k];
}

// The i-th of S sampled rows of n: one row of [i n / S, (i + 1) n / S), at a
// place within it that multiplicative hashing (Knuth) of i gives.  A fixed
// stride would miss whole groups of a base whose rows come in turns (24
// clusters in turn, stride 24: every row's threshold but one cluster's came
// from a foreign cluster, its list overflowed, and 100k x 64 took 160 ms
// instead of 10).
__device__ __forceinline__ int64_t sampled_row(int64_t i, int64_t S, int64_t n) {
  const int64_t lo = i * n / S, width = (i + 1) * n / S - lo;
  unsigned long long h = (unsigned long long)(i + 1) * 0x9e3779b97f4a7c15ull;
  h = (h ^ (h >> 32)) * 0x9e3779b97f4a7c15ull;
  return lo + (int64_t)(((h >> 32) * (unsigned long long)width) >> 32);
}

// Row i of dst = row rows[i] (or the i-th sampled row of `total`) of src, in
// 16-byte pieces: one warp per row.
__global__ void gather_split_rows(const uint4* __restrict__ src, int64_t pieces, const int64_t* __restrict__ rows,
                                  int64_t total, int64_t n, uint4* __restrict__ dst,
                                  const float* __restrict__ nrm, float* __restrict__ dnrm) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = warp; i < n; i += nwarps) {
    const int64_t r = rows ? rows[i] : sampled_row(i, n, total);
    for (int64_t c = lane; c < pieces; c += 32) dst[i * pieces + c] = __ldg(src + r * pieces + c);
    if (dnrm && lane == 0) dnrm[i] = nrm[r];
  }
}

__device__ __forceinline__ uint32_t float_key(float a) {  // order-preserving
  const uint32_t u = __float_as_uint(a);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// The threshold of each row: about its rank-th smallest approximate distance
// among the S sampled columns (dot products D[row][0..S)).  Any threshold is
// valid; its rank sets how many columns the pass over the base keeps.  One
// warp per row: every lane keeps the 8 smallest of its columns, and the
// rank-th smallest of those 256 is found bit by bit (a lane that holds more
// than 8 of the smallest only makes the threshold larger).
constexpr int kSampleKeep = 8;
__global__ void __launch_bounds__(256) sample_threshold(const float* __restrict__ D, int64_t S, int64_t m,
                                                        const float* __restrict__ qn,
                                                        const float* __restrict__ snrm, int rank,
                                                        float* __restrict__ tau) {
  const int lane = threadIdx.x & 31;
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (row >= m) return;
  const float q = qn[row];
  const float* d = D + row * S;
  float keep[kSampleKeep];
#pragma unroll
  for (int s = 0; s < kSampleKeep; ++s) keep[s] = INFINITY;
  constexpr int kAhead = 8;  // loads in flight per lane
  for (int64_t j0 = lane; j0 < S; j0 += 32 * kAhead) {
    float a[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      const int64_t j = j0 + 32 * u;
      a[u] = j < S ? __fmaf_rn(-2.0f, __ldg(d + j), __fadd_rn(q, __ldg(snrm + j))) : INFINITY;
    }
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      if (a[u] < keep[kSampleKeep - 1]) {
        float c = a[u];
#pragma unroll
        for (int s = 0; s < kSampleKeep; ++s) {
          const float lo = fminf(keep[s], c);
          c = fmaxf(keep[s], c);
          keep[s] = lo;
        }
      }
    }
  }
  uint32_t key[kSampleKeep], at = 0;
#pragma unroll
  for (int s = 0; s < kSampleKeep; ++s) key[s] = float_key(keep[s]);
  for (uint32_t bit = 0x80000000u; bit; bit >>= 1) {
    unsigned below = 0;
#pragma unroll
    for (int s = 0; s < kSampleKeep; ++s) below += key[s] < (at | bit) ? 1u : 0u;
    if (__reduce_add_sync(0xffffffffu, below) < (unsigned)rank) at |= bit;
  }
  if (lane == 0) tau[row] = key_float(at);
}

// Step 3: one warp per row and eight rows per block.  The R-th smallest
// approximate distance is found bit by bit; the columns up to it plus twice
// the error bound are the row's candidates.  The block then spreads all
// (row, candidate) pairs of its rows over its threads -- FP64 is the scarce
// unit here (1.25 TFLOP/s), and a warp per row would leave a second, nearly
// empty round for every row -- each summing in dimension order, and every
// warp sorts its row.
__global__ void __launch_bounds__(32 * kFinRows) finish_rows(
    const float* __restrict__ x, int d, int64_t r0, int64_t m, const KnnHit* __restrict__ list,
    const int* __restrict__ cnt, int cap, const float* __restrict__ tau, const double* __restrict__ nrm64,
    const unsigned long long* __restrict__ max_nrm, int R, int kmax, int32_t* __restrict__ out,
    int* __restrict__ failed) {
  extern __shared__ unsigned char sm_raw[];
  // per row: kmax distances, kmax ids, cap keys
  double* sd = reinterpret_cast<double*>(sm_raw);
  int* si = reinterpret_cast<int*>(sd + (size_t)kFinRows * kmax);
  uint32_t* keys = reinterpret_cast<uint32_t*>(si + (size_t)kFinRows * kmax);
  __shared__ int s_m[kFinRows];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t row = (int64_t)blockIdx.x * kFinRows + w;
  const int64_t gi = r0 + row;
  int* rid = si + (size_t)w * kmax;
  int take = 0;
  if (row < m) {
    const KnnHit* l = list + row * cap;
    uint32_t* rk = keys + (size_t)w * cap;
    const int n = cnt[row];
    bool ok = n <= cap;
    if (ok) {
      for (int i = lane; i < n; i += 32) rk[i] = l[i].col < 0 ? 0xffffffffu : float_key(l[i].a);
      __syncwarp();
      uint32_t at = 0;
      for (uint32_t bit = 0x80000000u; bit; bit >>= 1) {
        unsigned below = 0;
        for (int i = lane; i < n; i += 32) below += rk[i] < (at | bit) ? 1u : 0u;
        if (__reduce_add_sync(0xffffffffu, below) < (unsigned)R) at |= bit;
      }
      // the R-th smallest (all bits set if the list has fewer)
      const double err = approx_error(nrm64[gi], sqrt(__longlong_as_double((long long)*max_nrm)), d);
      const float bound = __double2float_ru((double)key_float(at) + 2.0 * err);
      ok = at != 0xffffffffu && bound < tau[row];
      if (ok) {
        const uint32_t kb = float_key(bound);
        for (int b = 0; b < n; b += 32) {
          const bool c = b + lane < n && rk[b + lane] <= kb;
          const unsigned mask = __ballot_sync(0xffffffffu, c);
          const int p = take + __popc(mask & ((1u << lane) - 1u));
          if (c && p < kmax) rid[p] = l[b + lane].col;
          take += __popc(mask);
        }
        ok = take >= R && take <= kmax;
      }
    }
    if (!ok) {
      take = 0;
      if (lane == 0) {
        out[gi * R] = -1;  // marks the row for step 4
        atomicAdd(failed, 1);
      }
    }
  }
  if (lane == 0) s_m[w] = take;
  __syncthreads();
  int total = 0;
  int off[kFinRows];
#pragma unroll
  for (int i = 0; i < kFinRows; ++i) {
    off[i] = total;
    total += s_m[i];
  }
  const bool vec = (d & 3) == 0 && ((uintptr_t)x & 15) == 0;
  for (int p = threadIdx.x; p < total; p += blockDim.x) {
    int r = 0, k = p;
#pragma unroll
    for (int i = 1; i < kFinRows; ++i)
      if (p >= off[i]) {
        r = i;
        k = p - off[i];
      }
    const float* q = x + (r0 + (int64_t)blockIdx.x * kFinRows + r) * d;
    const float* y = x + (int64_t)si[(size_t)r * kmax + k] * d;
    double s = 0.0;
    auto add = [&](double a, double b) {
      const double t = a - b;
      s = fma(t, t, s);
    };
    if (vec) {
#pragma unroll 4
      for (int c = 0; c < d; c += 4) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(y + c)), b = __ldg(reinterpret_cast<const float4*>(q + c));
        bool special = false;
        const double ax = widen(a.x, special), ay = widen(a.y, special), az = widen(a.z, special), aw = widen(a.w, special);
        const double bx = widen(b.x, special), by = widen(b.y, special), bz = widen(b.z, special), bw = widen(b.w, special);
        if (special) {
          add((double)a.x, (double)b.x);
          add((double)a.y, (double)b.y);
          add((double)a.z, (double)b.z);
          add((double)a.w, (double)b.w);
        } else {
          add(ax, bx);
          add(ay, by);
          add(az, bz);
          add(aw, bw);
        }
      }
    } else {
      for (int c = 0; c < d; ++c) add((double)__ldg(y + c), (double)__ldg(q + c));
    }
    sd[(size_t)r * kmax + k] = s;
  }
  __syncthreads();
  if (take == 0) return;
  double* rd = sd + (size_t)w * kmax;
  int np2 = 2;
  while (np2 < take) np2 <<= 1;  // at most kmax, a power of two
  for (int i = take + lane; i < np2; i += 32) {
    rd[i] = INFINITY;
    rid[i] = INT32_MAX;
  }
  __syncwarp();
  for (int step = 2; step <= np2; step <<= 1)
    for (int sub = step >> 1; sub >= 1; sub >>= 1) {
      for (int t = lane; t < np2 / 2; t += 32) {
        const int i = 2 * t - (t & (sub - 1)), j = i + sub;
        const bool up = (i & step) == 0;
        const bool sw = up ? key_less64(rd[j], rid[j], rd[i], rid[i]) : key_less64(rd[i], rid[i], rd[j], rid[j]);
        if (sw) {
          const double a = rd[i];
          rd[i] = rd[j];
          rd[j] = a;
          const int u = rid[i];
          rid[i] = rid[j];
          rid[j] = u;
        }
      }
      __syncwarp();
    }
  for (int k = lane; k < R; k += 32) out[gi * R + k] = rid[k];
}

// Step 4 on the rows in `rows` (host, ascending): their dot products with the
// whole base in memory, K candidates, then 1024 for those that need them.  A
// block of dot products of more than the stream-ordered pool keeps mapped (it
// takes up to 8 GB) is allocated apart: 200k x 64, degree 129, 350 ms from the
// pool, which maps it anew in every call, and 342 ms.
rte_status stored_rows(const float* x, int64_t n, int d, int dp, int degree, const uint16_t* A, const uint16_t* B,
                       const float* n32, const double* n64, const unsigned long long* max_nrm,
                       const std::vector<int64_t>& rows, int32_t* g, int* err, int64_t& n_retried, cudaStream_t st) {
  const int K = std::min<int64_t>(std::min(2 * degree + 32, kSelPool), n);
  const int Kp = 1 << (int)std::ceil(std::log2((double)std::max(K, 2)));
  const int K2 = (int)std::min<int64_t>(kMaxCand, n);
  // rows per block: the FP32 dot-product block stays under 8 GB
  int64_t mb = std::max<int64_t>(128, std::min<int64_t>(8192, (int64_t)(8ll << 30) / (n * 4)));
  mb = std::min<int64_t>(mb, (int64_t)rows.size());
  const int64_t pieces = 3 * (int64_t)dp * 2 / 16;
  DevBuf<float> apart;
  AsyncBuf pooled, Af, cand, excl, drows, drr, loc, fl;
  if ((size_t)mb * n * 4 > kScratchKeepBytes)
    RTE_CUDA(apart.alloc((size_t)mb * n));
  else
    RTE_CUDA(pooled.alloc((size_t)mb * n * 4, st));
  float* const D = apart.p ? apart.p : pooled.as<float>();
  RTE_CUDA(Af.alloc((size_t)mb * 3 * dp * 2, st));
  RTE_CUDA(cand.alloc((size_t)mb * kMaxCand * 4, st));
  RTE_CUDA(excl.alloc((size_t)mb * 4, st));
  RTE_CUDA(drows.alloc((size_t)mb * 8, st));
  RTE_CUDA(drr.alloc((size_t)mb * 8, st));
  RTE_CUDA(loc.alloc((size_t)mb * 4, st));
  RTE_CUDA(fl.alloc(4, st));
  std::vector<int64_t> rrows;
  std::vector<int32_t> hfirst, rlocal;
  for (size_t b0 = 0; b0 < rows.size(); b0 += (size_t)mb) {
    const int64_t m = std::min<int64_t>(mb, (int64_t)(rows.size() - b0));
    RTE_CUDA(cudaMemcpyAsync(drows.p, rows.data() + b0, m * 8, cudaMemcpyHostToDevice, st));
    GemmArgs ga{};
    if (rows[b0 + m - 1] - rows[b0] == m - 1) {  // rows that follow one another: in place
      ga.A = A + rows[b0] * 3 * dp;
    } else {
      gather_split_rows<<<(unsigned)std::min<int64_t>((m + 7) / 8, 4096), 256, 0, st>>>(
          reinterpret_cast<const uint4*>(A), pieces, drows.as<int64_t>(), 0, m, Af.as<uint4>(), nullptr, nullptr);
      ga.A = Af.p;
    }
    ga.B = B;
    ga.M = (int)m;
    ga.N = (int)n;
    ga.K = 3 * dp;
    ga.epilogue = kEpiStoreF32;
    ga.C = D;
    ga.ldc = (int)n;
    ga.err = err;
    RTE_CUDA(gemm_bf16_tn(ga, st));
    select_rows<<<(unsigned)m, kSelThreads, 0, st>>>(D, n, drows.as<int64_t>(), n, n32, K, nullptr,
                                                       cand.as<int32_t>(), excl.as<float>());
    RTE_CUDA(cudaGetLastError());
    RTE_CUDA(cudaMemsetAsync(fl.p, 0, 4, st));
    rerank_rows<<<(unsigned)m, 256, (size_t)Kp * 12, st>>>(x, d, drows.as<int64_t>(), cand.as<int32_t>(), K, Kp,
                                                 excl.as<float>(), n64, max_nrm, degree, g, fl.as<int>());
    RTE_CUDA(cudaGetLastError());
    int nfail = 0;
    RTE_CUDA(cudaMemcpyAsync(&nfail, fl.p, 4, cudaMemcpyDeviceToHost, st));
    RTE_CUDA(cudaStreamSynchronize(st));
    if (!nfail) continue;
    // rows not certified (first entry -1): K2 candidates from the same
    // block of dot products, which the next block's GEMM has not yet
    // overwritten (same stream)
    rrows.clear();
    rlocal.clear();
    // the first entries of every row between the block's first and last
    // (the rows ascend)
    const int64_t lo = rows[b0], span = rows[b0 + m - 1] - lo + 1;
    hfirst.resize((size_t)span);
    RTE_CUDA(cudaMemcpy2DAsync(hfirst.data(), 4, g + lo * degree, (size_t)degree * 4, 4, (size_t)span,
                               cudaMemcpyDeviceToHost, st));
    RTE_CUDA(cudaStreamSynchronize(st));
    for (int64_t i = 0; i < m; ++i)
      if (hfirst[rows[b0 + i] - lo] < 0) {
        rrows.push_back(rows[b0 + i]);
        rlocal.push_back((int32_t)i);
      }
    const int64_t mr = (int64_t)rrows.size();
    n_retried += mr;
    RTE_CUDA(cudaMemcpyAsync(loc.p, rlocal.data(), mr * 4, cudaMemcpyHostToDevice, st));
    RTE_CUDA(cudaMemcpyAsync(drr.p, rrows.data(), mr * 8, cudaMemcpyHostToDevice, st));
    select_rows<<<(unsigned)mr, kSelThreads, 0, st>>>(D, n, drows.as<int64_t>(), n, n32, K2,
                                                        loc.as<int32_t>(), cand.as<int32_t>(), excl.as<float>());
    RTE_CUDA(cudaGetLastError());
    RTE_CUDA(cudaMemsetAsync(fl.p, 0, 4, st));
    rerank_rows<<<(unsigned)mr, 256, (size_t)kMaxCand * 12, st>>>(
        x, d, drr.as<int64_t>(), cand.as<int32_t>(), K2, kMaxCand, excl.as<float>(), n64, max_nrm, degree, g,
        fl.as<int>());
    RTE_CUDA(cudaGetLastError());
    RTE_CUDA(cudaMemcpyAsync(&nfail, fl.p, 4, cudaMemcpyDeviceToHost, st));
    RTE_CUDA(cudaStreamSynchronize(st));
    if (nfail) return fail(RTE_EIO, "kNN graph: " + std::to_string(nfail) + " rows could not be certified exact");
  }
  return RTE_OK;
}

}  // namespace
}  // namespace rte

using namespace rte;

extern "C" rte_status rte_knn_graph_plan(int64_t n, int degree, int64_t* plan) {
  clear_error();
  if (!plan) return fail(RTE_EINVAL, "NULL argument");
  if (n <= 0 || n >= INT32_MAX || degree <= 0 || degree > 256 || n <= degree)
    return fail(RTE_EINVAL, "degree must be in [1, min(256, n - 1)]");
  const FilterPlan p = filter_plan(n, degree);
  plan[0] = p.use;
  plan[1] = p.sample;
  plan[2] = p.rank;
  plan[3] = p.cap;
  plan[4] = p.block;
  plan[5] = p.use ? (int64_t)finish_smem(p.cap, p.kmax) : 0;
  return RTE_OK;
}

extern "C" rte_status rte_knn_graph(const float* base, int64_t n, int d, int degree, int device,
                                    int32_t* graph, void* stream) {
  clear_error();
  if (!base || !graph || n <= 0 || d <= 0) return fail(RTE_EINVAL, "bad kNN graph arguments");
  if (degree <= 0 || degree > 256 || n <= degree) return fail(RTE_EINVAL, "degree must be in [1, min(256, n - 1)]");
  if (n >= INT32_MAX) return fail(RTE_EINVAL, "n must be below 2^31");
  DeviceGuard guard(device);
  cudaStream_t st = (cudaStream_t)stream;
  const int dp = (d + 7) & ~7;
  AsyncBuf xd, A, B, n32, n64, outd, part, mu, flags;
  const bool base_dev = is_device_ptr(base), graph_dev = is_device_ptr(graph);
  const float* x = base;
  if (!base_dev) {
    RTE_CUDA(xd.alloc((size_t)n * d * 4, st));
    RTE_CUDA(cudaMemcpyAsync(xd.p, base, (size_t)n * d * 4, cudaMemcpyHostToDevice, st));
    x = xd.as<float>();
  }
  RTE_CUDA(A.alloc((size_t)n * 3 * dp * 2, st));
  RTE_CUDA(B.alloc((size_t)n * 3 * dp * 2, st));
  RTE_CUDA(n32.alloc((size_t)n * 4, st));
  RTE_CUDA(n64.alloc((size_t)n * 8, st));
  int32_t* g = graph;
  if (!graph_dev) {
    RTE_CUDA(outd.alloc((size_t)n * degree * 4, st));
    g = outd.as<int32_t>();
  }
  RTE_CUDA(part.alloc((size_t)kMeanSlices * d * 8, st));
  RTE_CUDA(mu.alloc((size_t)d * 4, st));
  // the largest squared norm, the pipeline's error word, rows not certified
  RTE_CUDA(flags.alloc(16, st));
  RTE_CUDA(cudaMemsetAsync(flags.p, 0, 16, st));
  unsigned long long* max_nrm = flags.as<unsigned long long>();
  int* err = flags.as<int>() + 2;
  int* nfail = flags.as<int>() + 3;
  col_sum_slices<<<dim3((unsigned)((d + 127) / 128), kMeanSlices), 128, 0, st>>>(x, n, d, part.as<double>());
  col_mean_finish<<<(unsigned)((d + 127) / 128), 128, 0, st>>>(part.as<double>(), n, d, mu.as<float>());
  split_rows<<<(unsigned)std::min<int64_t>((n + 7) / 8, 65535), 256, 0, st>>>(
      x, mu.as<float>(), n, d, dp, A.as<__nv_bfloat16>(), B.as<__nv_bfloat16>(), n32.as<float>(),
      n64.as<double>(), max_nrm);
  RTE_CUDA(cudaGetLastError());
  std::vector<int64_t> left;  // rows for step 4
  const FilterPlan fp = filter_plan(n, degree);
  if (fp.use) {
    const int64_t S = fp.sample, mb = fp.block;
    const int cap = fp.cap, kmax = fp.kmax;
    AsyncBuf Bs, ns, D, tau, cnt, list;
    RTE_CUDA(Bs.alloc((size_t)S * 3 * dp * 2, st));
    RTE_CUDA(ns.alloc((size_t)S * 4, st));
    RTE_CUDA(D.alloc((size_t)mb * S * 4, st));
    RTE_CUDA(tau.alloc((size_t)mb * 4, st));
    RTE_CUDA(cnt.alloc((size_t)mb * 4, st));
    RTE_CUDA(list.alloc((size_t)mb * cap * sizeof(KnnHit), st));
    gather_split_rows<<<(unsigned)std::min<int64_t>((S + 7) / 8, 4096), 256, 0, st>>>(
        B.as<uint4>(), 3 * (int64_t)dp * 2 / 16, nullptr, n, S, Bs.as<uint4>(), n32.as<float>(),
        ns.as<float>());
    RTE_CUDA(cudaGetLastError());
    const size_t fin_smem = finish_smem(cap, kmax);
    // the same limit in every call: it belongs to the kernel, and a build of a
    // smaller degree on another thread must not lower it under this one
    RTE_CUDA(cudaFuncSetAttribute(finish_rows, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)finish_smem(kMaxCap, kMaxFinish)));
    for (int64_t r0 = 0; r0 < n; r0 += mb) {
      const int64_t m = std::min(mb, n - r0);
      const uint16_t* Ar = A.as<uint16_t>() + r0 * 3 * dp;
      GemmArgs ga{};
      ga.A = Ar;
      ga.B = Bs.p;
      ga.M = (int)m;
      ga.N = (int)S;
      ga.K = 3 * dp;
      ga.epilogue = kEpiStoreF32;
      ga.C = D.p;
      ga.ldc = (int)S;
      ga.err = err;
      RTE_CUDA(gemm_bf16_tn(ga, st));
      sample_threshold<<<(unsigned)((m + 7) / 8), 256, 0, st>>>(D.as<float>(), S, m, n32.as<float>() + r0,
                                                                ns.as<float>(), fp.rank, tau.as<float>());
      RTE_CUDA(cudaGetLastError());
      RTE_CUDA(cudaMemsetAsync(cnt.p, 0, (size_t)m * 4, st));
      KnnFilterArgs f{};
      f.A = Ar;
      f.B = B.p;
      f.M = (int)m;
      f.N = (int)n;
      f.K = 3 * dp;
      f.r0 = r0;
      f.qn = n32.as<float>() + r0;
      f.nrm = n32.as<float>();
      f.tau = tau.as<float>();
      f.list = list.as<KnnHit>();
      f.cnt = cnt.as<int>();
      f.cap = cap;
      f.err = err;
      RTE_CUDA(knn_filter(f, st));
      finish_rows<<<(unsigned)((m + kFinRows - 1) / kFinRows), 32 * kFinRows, fin_smem, st>>>(
          x, d, r0, m, f.list, f.cnt, cap, f.tau, n64.as<double>(), max_nrm, degree, kmax, g, nfail);
      RTE_CUDA(cudaGetLastError());
    }
    int hf[2] = {0, 0};  // error word, rows not certified
    RTE_CUDA(cudaMemcpyAsync(hf, err, 8, cudaMemcpyDeviceToHost, st));
    RTE_CUDA(cudaStreamSynchronize(st));
    if (hf[0]) return fail(RTE_ETIMEOUT, "GEMM pipeline wait ran out (code " + std::to_string(hf[0]) + ")");
    if (hf[1]) {
      std::vector<int32_t> first((size_t)n);
      RTE_CUDA(cudaMemcpy2DAsync(first.data(), 4, g, (size_t)degree * 4, 4, (size_t)n, cudaMemcpyDeviceToHost, st));
      RTE_CUDA(cudaStreamSynchronize(st));
      for (int64_t i = 0; i < n; ++i)
        if (first[i] < 0) left.push_back(i);
    }
  } else {
    left.resize((size_t)n);
    for (int64_t i = 0; i < n; ++i) left[i] = i;
  }
  int64_t n_retried = 0;
  if (!left.empty()) {
    const rte_status s = stored_rows(x, n, d, dp, degree, A.as<uint16_t>(), B.as<uint16_t>(), n32.as<float>(),
                                     n64.as<double>(), max_nrm, left, g, err, n_retried, st);
    if (s != RTE_OK) return s;
  }
  if (getenv("RTE_KNN_VERBOSE"))
    fprintf(stderr, "rte_knn_graph: n %lld d %d degree %d: %lld rows in memory, %lld rows retried with %d candidates\n",
            (long long)n, d, degree, (long long)left.size(), (long long)n_retried, (int)std::min<int64_t>(kMaxCand, n));
  int herr = 0;
  RTE_CUDA(cudaMemcpyAsync(&herr, err, 4, cudaMemcpyDeviceToHost, st));
  if (!graph_dev) RTE_CUDA(cudaMemcpyAsync(graph, g, (size_t)n * degree * 4, cudaMemcpyDeviceToHost, st));
  RTE_CUDA(cudaStreamSynchronize(st));
  if (herr) return fail(RTE_ETIMEOUT, "GEMM pipeline wait ran out (code " + std::to_string(herr) + ")");
  return RTE_OK;
}
