// knn_filter.cu -- see knn_filter.h.
//
// The same pipeline as gemm_bf16_tn_kernel (gemm_tc.cu): a persistent grid of
// one CTA per SM over contiguous ranges of output tiles, row-block major; one
// warp streams 64-wide K chunks with TMA (128-byte swizzle), one issues
// tcgen05.mma (M = 128, N = 256, K = 16) into one of two 256-column TMEM
// accumulators, and 16 warps read them back.  What differs is the end: the
// epilogue forms each approximate distance, compares it with its row's
// threshold and appends the few below it to the row's list.
//
// Why: writing the dot products (4 n^2 bytes) and reading them back to select
// from cost more than the products.  On one GB300 a 100k x 128 degree-32
// graph took 105 ms with the products stored and sorted, 11.5 ms
// with this pass (its kernel: 6.9 ms for 7.7 TFLOP).
//
// What bounds it: with K <= 384 (d <= 128) the row block's A chunks stay in
// shared memory and only B streams: 196 KB per 128 x 256 tile instead of
// 295 KB (and 196 KB per 128 x 128 tile in the stored form), 8.7 TB/s from L2
// at the measured rate.  16384 x 100k x 128 takes 1.13 ms, 1.12 PFLOP/s: the
// tensor pipe is active 49 % of the time, the epilogue keeps issue at 49 %,
// DRAM is at 12 % and L2's sectors at 30 % of their peaks.  No unit is
// saturated: a tile waits for its operands and for its epilogue's handoff.
//
// A list slot is reserved with an atomic on the row's counter, eight at a
// time per thread: a thread meets a hit in one tile of three, and one atomic
// per hit would cost its warp an L2 round trip each.
#include <cuda.h>
#include <cuda_runtime.h>

#include <atomic>

#include "knn_filter.h"
#include "tc_common.cuh"

namespace rte {

namespace {

using namespace tc;

constexpr int BM = 128, BN = 256, BK = 64;
constexpr int A_BYTES = BM * BK * 2;
constexpr int B_BYTES = BN * BK * 2;
constexpr int kResidentChunks = 6;
constexpr int kStages = 4;  // resident: 6 A chunks + 4 of B; streamed: 4 of A + B
constexpr int RING_BYTES = kResidentChunks * A_BYTES + kStages * B_BYTES;
static_assert(kStages * (A_BYTES + B_BYTES) <= RING_BYTES, "streamed stages fit");
constexpr int kEpiWarps = 16;
constexpr int kCols = BN / (kEpiWarps / 4);  // columns per epilogue warp and tile
constexpr int kProducerWarp = kEpiWarps, kMmaWarp = kEpiWarps + 1;
constexpr int kThreads = 32 * (kEpiWarps + 2);
constexpr int kBars = 2 * kStages + 7;
constexpr int SMEM_BYTES = RING_BYTES + 1024 /*align*/ + 8 * kBars + 16;
constexpr int kReserve = 8;
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) |
                            ((uint32_t)(BM >> 4) << 24);

__global__ void __launch_bounds__(kThreads, 1)
    knn_filter_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      KnnFilterArgs g) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + RING_BYTES);
  const uint32_t full0 = smem_u32(bars), empty0 = smem_u32(bars + kStages);
  const uint32_t tfull0 = smem_u32(bars + 2 * kStages), tempty0 = smem_u32(bars + 2 * kStages + 2);
  const uint32_t afull = smem_u32(bars + 2 * kStages + 4);
  const uint32_t afree = smem_u32(bars + 2 * kStages + 5);
  const uint32_t drain = smem_u32(bars + 2 * kStages + 6);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kBars);
  __shared__ int s_abort;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nk = (g.K + BK - 1) / BK;
  const int n_tiles = (g.N + BN - 1) / BN;
  const int m_tiles = (g.M + BM - 1) / BM;
  const bool resident = nk <= kResidentChunks;
  const long long total = (long long)m_tiles * n_tiles;
  const long long t_begin = total * blockIdx.x / gridDim.x;
  const long long t_end = total * (blockIdx.x + 1) / gridDim.x;
  auto a_addr = [&](int s, int kt) -> uint8_t* { return resident ? ring + kt * A_BYTES : ring + s * (A_BYTES + B_BYTES); };
  auto b_addr = [&](int s) -> uint8_t* {
    return resident ? ring + kResidentChunks * A_BYTES + s * B_BYTES : ring + s * (A_BYTES + B_BYTES) + A_BYTES;
  };

  if (threadIdx.x == 0) {
    s_abort = 0;
    for (int i = 0; i < kStages; ++i) {
      mbar_init(full0 + 8 * i, 1);
      mbar_init(empty0 + 8 * i, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(tfull0 + 8 * a, 1);
      mbar_init(tempty0 + 8 * a, kEpiWarps * 32);
    }
    mbar_init(afull, 1);
    mbar_init(afree, 1);
    mbar_init(drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(2 * BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  int* abort = &s_abort;

  if (warp == kProducerWarp) {
    if (lane == 0) {
      int issued = 0, a_loads = 0, cur_mt = -1;
      bool ok = true;
      for (long long ti = t_begin; ti < t_end && ok; ++ti) {
        const int mt = (int)(ti / n_tiles), nt = (int)(ti % n_tiles);
        if (resident && mt != cur_mt) {
          // a new row block: wait until the MMAs are done with the old one
          if (a_loads > 0 && !mbar_wait(afree, (a_loads - 1) & 1, g.err, 6, abort, g.wait_limit)) {
            ok = false;
            break;
          }
          mbar_expect_tx(afull, (uint32_t)(nk * A_BYTES));
          for (int kt = 0; kt < nk; ++kt) tma_load_2d(smem_u32(a_addr(0, kt)), &tmA, kt * BK, mt * BM, afull);
          ++a_loads;
          cur_mt = mt;
        }
        for (int kt = 0; kt < nk; ++kt) {
          const int s = issued % kStages, r = issued / kStages;
          if (issued >= kStages && !mbar_wait(empty0 + 8 * s, (r - 1) & 1, g.err, 1, abort, g.wait_limit)) {
            ok = false;
            break;
          }
          if (*(volatile int*)abort) {
            ok = false;
            break;
          }
          mbar_expect_tx(full0 + 8 * s, resident ? B_BYTES : A_BYTES + B_BYTES);
          if (!resident) tma_load_2d(smem_u32(a_addr(s, kt)), &tmA, kt * BK, mt * BM, full0 + 8 * s);
          tma_load_2d(smem_u32(b_addr(s)), &tmB, kt * BK, nt * BN, full0 + 8 * s);
          ++issued;
        }
      }
      if (!ok) *(volatile int*)abort = 1;
      // let every copy in flight land before the CTA can exit
      for (int i = (issued > kStages ? issued - kStages : 0); i < issued; ++i)
        mbar_wait(full0 + 8 * (i % kStages), (i / kStages) & 1, g.err, 2);
      if (a_loads > 0) mbar_wait(afull, (a_loads - 1) & 1, g.err, 2);
    }
  } else if (warp == kMmaWarp) {
    if (lane == 0) {
      bool ok = true;
      int used = 0, t = 0, a_uses = 0, cur_mt = -1;
      for (long long ti = t_begin; ti < t_end && ok; ++ti, ++t) {
        const int mt = (int)(ti / n_tiles);
        if (resident && mt != cur_mt) {
          if (cur_mt >= 0) mma_commit(afree);  // arrives once the MMAs on the old block finish
          if (!mbar_wait(afull, a_uses & 1, g.err, 3, abort, g.wait_limit)) {
            ok = false;
            break;
          }
          ++a_uses;
          cur_mt = mt;
        }
        const int a = t & 1;
        if (t >= 2 && !mbar_wait(tempty0 + 8 * a, ((t >> 1) - 1) & 1, g.err, 5, abort, g.wait_limit)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t d = tmem + (uint32_t)(a * BN);
        for (int kt = 0; kt < nk; ++kt, ++used) {
          const int s = used % kStages, r = used / kStages;
          if (!mbar_wait(full0 + 8 * s, r & 1, g.err, 3, abort, g.wait_limit)) {
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t ad = sw128_desc(smem_u32(a_addr(s, kt)));
          const uint64_t bd = sw128_desc(smem_u32(b_addr(s)));
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk)
            mma_bf16(d, ad + (uint64_t)(2 * kk), bd + (uint64_t)(2 * kk), kIdesc, (kt | kk) != 0);
          mma_commit(empty0 + 8 * s);
        }
        if (!ok) break;
        mma_commit(tfull0 + 8 * a);
      }
      if (!ok) *(volatile int*)abort = 1;
      // no MMA may still run when TMEM is freed, whatever path led here
      mma_commit(drain);
      mbar_wait(drain, 0, g.err, 7);
    }
  } else {
    // warp w owns accumulator rows 32 (w % 4) .. +31 (one per lane) and
    // columns kCols * (w / 4) .. of every tile
    const int quarter = warp & 3, part = warp >> 2;
    const int row_l = quarter * 32 + lane;
    int cur_mt = -1, row = 0, pos = 0, lim = 0, self = -1;
    float qn = 0.0f, tau = 0.0f;
    KnnHit* out = nullptr;
    auto append = [&](float a, int col) {
      if (pos == lim) {
        pos = atomicAdd(g.cnt + row, kReserve);
        lim = pos + kReserve;
      }
      if (pos < g.cap) out[pos] = KnnHit{a, col};
      ++pos;
    };
    auto finish_row = [&]() {  // slots reserved and not used
      for (; pos < lim; ++pos)
        if (pos < g.cap) out[pos] = KnnHit{__int_as_float(0x7f800000), -1};
      pos = lim = 0;
    };
    int t = 0;
    for (long long ti = t_begin; ti < t_end; ++ti, ++t) {
      const int mt = (int)(ti / n_tiles), nt = (int)(ti % n_tiles);
      if (mt != cur_mt) {
        if (cur_mt >= 0) finish_row();
        cur_mt = mt;
        row = mt * BM + row_l;
        const bool live = row < g.M;
        qn = live ? __ldg(g.qn + row) : 0.0f;
        tau = live ? __ldg(g.tau + row) : -__int_as_float(0x7f800000);
        self = live ? (int)(g.r0 + row) : -1;
        out = g.list + (size_t)(live ? row : 0) * g.cap;
      }
      const int a = t & 1;
      const bool ok = __all_sync(0xffffffffu, mbar_wait(tfull0 + 8 * a, (t >> 1) & 1, g.err, 4, abort, g.wait_limit));
      if (!ok) {
        *(volatile int*)abort = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int n0 = nt * BN + part * kCols;
      const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(a * BN + part * kCols);
#pragma unroll 1
      for (int c0 = 0; c0 < kCols; c0 += 32) {
        uint32_t r[32];
        __syncwarp();  // lanes that appended rejoin before the collective load
        tmem_ld32(taddr + (uint32_t)c0, r);
        float nv[32];
        const int col0 = n0 + c0;
        if (col0 + 32 <= g.N) {
#pragma unroll
          for (int i = 0; i < 32; i += 4) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(g.nrm + col0 + i));
            nv[i] = v.x;
            nv[i + 1] = v.y;
            nv[i + 2] = v.z;
            nv[i + 3] = v.w;
          }
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i)  // columns past the end are never below a threshold
            nv[i] = col0 + i < g.N ? __ldg(g.nrm + col0 + i) : __int_as_float(0x7f800000);
        }
        tmem_wait_ld();
        if (c0 + 32 == kCols) {  // accumulator drained: hand it back to the MMA issuer
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          mbar_arrive(tempty0 + 8 * a);
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const float d = __fmaf_rn(-2.0f, __uint_as_float(r[i]), __fadd_rn(qn, nv[i]));
          if (d < tau && col0 + i != self) append(d, col0 + i);
        }
      }
    }
    if (cur_mt >= 0) finish_row();
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN));
  }
}

}  // namespace

cudaError_t knn_filter(const KnnFilterArgs& g, cudaStream_t st) {
  if (g.M <= 0 || g.N <= 0 || g.K <= 0 || (g.K & 7) || !g.A || !g.B || !g.list || !g.cnt || g.cap <= 0)
    return cudaErrorInvalidValue;
  if (((uintptr_t)g.A & 15) || ((uintptr_t)g.B & 15) || ((uintptr_t)g.nrm & 15)) return cudaErrorInvalidValue;
  CUtensorMap ma, mb;
  if (!make_map_bf16(&ma, g.A, g.M, g.K, BK, BM) || !make_map_bf16(&mb, g.B, g.N, g.K, BK, BN))
    return cudaErrorNotSupported;
  int dev = 0, sms = 1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return cudaErrorInvalidDevice;
  static std::atomic<bool> attr[64];
  if (!attr[dev].load(std::memory_order_acquire)) {
    const cudaError_t e =
        cudaFuncSetAttribute(knn_filter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) return e;
    attr[dev].store(true, std::memory_order_release);
  }
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 1;
  const long long tiles = (long long)((g.M + BM - 1) / BM) * ((g.N + BN - 1) / BN);
  KnnFilterArgs ga = g;
  ga.wait_limit = wait_limit();
  knn_filter_kernel<<<(unsigned)(tiles < sms ? tiles : sms), kThreads, SMEM_BYTES, st>>>(ma, mb, ga);
  return cudaGetLastError();
}

}  // namespace rte
