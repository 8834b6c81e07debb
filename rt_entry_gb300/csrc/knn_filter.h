// knn_filter.h -- the kNN builder's tensor-core pass: dot products of a block
// of rows against the whole base, of which only the columns whose approximate
// distance lies below the row's threshold leave the SM.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace rte {

struct KnnHit {
  float a;      // approximate distance |x|^2 + |y|^2 - 2 x.y
  int32_t col;  // base row, or -1: a slot reserved and not used
};

struct KnnFilterArgs {
  const void* A;       // BF16 [M][K], rows r0 .. r0+M-1 of the split base
  const void* B;       // BF16 [N][K]
  int M, N, K;
  int64_t r0;          // first row's index in the base (it is not its own neighbour)
  const float* qn;     // [M] squared norms of the rows
  const float* nrm;    // [N] squared norms of the base, 16-byte aligned
  const float* tau;    // [M] thresholds: every column with a < tau is kept
  KnnHit* list;        // [M][cap]
  int* cnt;            // [M] slots reserved per row, zero on entry (more than cap: overflow)
  int cap;
  int* err;
  long long wait_limit;  // set by knn_filter
};

// cudaErrorInvalidValue for unsupported shapes (K a multiple of 8, operands
// 16-byte aligned), cudaErrorNotSupported without a tensor-map encoder.
cudaError_t knn_filter(const KnnFilterArgs& a, cudaStream_t st);

}  // namespace rte
