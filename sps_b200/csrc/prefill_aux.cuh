// Small kernels around the prefill path: the document pre-pass and the visibility test hook.
#pragma once

#include "common.cuh"
#include "mask.cuh"

namespace spsattn {

__device__ __forceinline__ long long load_doc(const void* docs, int is_i64, size_t off) {
  return is_i64 ? reinterpret_cast<const long long*>(docs)[off]
                : (long long)reinterpret_cast<const int*>(docs)[off];
}

// One block per batch row: lo[b][i] = first row of the run of equal ids containing row i
// (inclusive max-scan of run-start positions), mono[b] = 1 iff the ids never decrease.
// Each thread scans kItems consecutive rows, so rows up to 8192 need a single pass.
__global__ void __launch_bounds__(1024)
doc_prepass_kernel(const void* docs, int is_i64, int64_t stride_b, int64_t stride_t, int N,
                   int* __restrict__ lo, int* __restrict__ mono, int* __restrict__ work_counter) {
  constexpr int kItems = 8;
  __shared__ int s_warp[32];
  __shared__ int s_carry;
  __shared__ int s_mono;
  const int b = blockIdx.x;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  // the attention kernel behind this one may be launched as a programmatic dependent: let its
  // blocks take the free SMs now (it waits for this grid before it reads lo / mono)
  grid_launch_dependents();
  const uint8_t* base =
      reinterpret_cast<const uint8_t*>(docs) + (size_t)b * stride_b * (is_i64 ? 8 : 4);
  if (tid == 0) {
    s_carry = 0;
    s_mono = 1;
    // the attention kernel that follows in the stream draws its work items from this counter
    if (b == 0 && work_counter != nullptr) *work_counter = 0;
  }
  __syncthreads();
  bool dec = false;
  for (int c0 = 0; c0 < N; c0 += 1024 * kItems) {
    const int i0 = c0 + tid * kItems;
    int v[kItems];
    long long prev = 0;
    if (i0 > 0 && i0 - 1 < N) prev = load_doc(base, is_i64, (size_t)(i0 - 1) * stride_t);
    int run = 0;
#pragma unroll
    for (int x = 0; x < kItems; ++x) {
      const int i = i0 + x;
      if (i < N) {
        const long long d = load_doc(base, is_i64, (size_t)i * stride_t);
        if (i > 0) {
          if (d != prev) run = i;
          dec |= d < prev;
        }
        prev = d;
      }
      v[x] = run;   // inclusive max of the run starts inside this thread's span
    }
    int tot = run;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, tot, o);
      if (lane >= o) tot = max(tot, u);
    }
    if (lane == 31) s_warp[warp] = tot;
    __syncthreads();
    if (warp == 0) {
      int wv = s_warp[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, wv, o);
        if (lane >= o) wv = max(wv, u);
      }
      s_warp[lane] = wv;
    }
    __syncthreads();
    int pre = __shfl_up_sync(0xffffffffu, tot, 1);   // everything before this thread in its warp
    if (lane == 0) pre = 0;
    pre = max(pre, max(s_carry, warp > 0 ? s_warp[warp - 1] : 0));
#pragma unroll
    for (int x = 0; x < kItems; ++x)
      if (i0 + x < N) lo[(size_t)b * N + i0 + x] = max(v[x], pre);
    __syncthreads();
    if (tid == 1023) s_carry = max(tot, pre);
    __syncthreads();
  }
  if (dec) s_mono = 0;
  __syncthreads();
  if (tid == 0) mono[b] = s_mono;
}

// Test hook for the bounded waits: one warp waits, with the given limit, on an mbarrier that
// nobody ever arrives at.  No copy or tensor-core operation is in flight; the wait gives up,
// reports SPSATTN_STATUS_WAIT_EXPIRED through the status word exactly as the attention kernels
// do, and the block ends normally.  result[0] = 1 when the wait returned "gave up".
__global__ void __launch_bounds__(32)
wait_expiry_kernel(int* status, unsigned long long limit_ns, int* result) {
  __shared__ __align__(8) unsigned long long s_bar;
  __shared__ int s_abort;
  const uint32_t bar = smem_u32(&s_bar);
  if (threadIdx.x == 0) {
    s_abort = 0;
    mbar_init(bar, 1);
    fence_barrier_init();
  }
  __syncwarp();
  bool ok = mbar_try_wait(bar, 0);
  if (!ok) ok = mbar_wait_slow(bar, 0, &s_abort, status, limit_ns);
  ok = __all_sync(0xffffffffu, ok);
  if (threadIdx.x == 0 && result != nullptr) result[0] = ok ? 0 : 1;
}

// vis[b][i][j] = 1 iff key row j is visible to query row i, using the kernels' own arithmetic.
__global__ void visibility_kernel(uint8_t* __restrict__ vis, const void* docs, int is_i64,
                                  int64_t stride_b, int64_t stride_t, const int* __restrict__ lo,
                                  const int* __restrict__ mono, int N, MaskParams m) {
  const int b = blockIdx.z;
  const int i = blockIdx.y;
  const uint8_t* base = docs == nullptr ? nullptr
                                         : reinterpret_cast<const uint8_t*>(docs) +
                                               (size_t)b * stride_b * (is_i64 ? 8 : 4);
  const bool general = docs != nullptr && mono[b] == 0;
  const int lo_i = (docs != nullptr && !general) ? lo[(size_t)b * N + i] : 0;
  int kmin[2], kmax[2];
  row_interval(m, i, lo_i, 0, kmin[0], kmax[0]);
  row_interval(m, i, lo_i, 1, kmin[1], kmax[1]);
  const long long my_doc = general ? load_doc(base, is_i64, (size_t)i * stride_t) : 0;
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < N; j += gridDim.x * blockDim.x) {
    const int p = m.ks == 2 ? (j & 1) : 0;
    const int kt = m.ks == 2 ? (j >> 1) : j;
    bool v = kt >= kmin[p] && kt <= kmax[p];
    if (v && general) v = load_doc(base, is_i64, (size_t)j * stride_t) == my_doc;
    vis[((size_t)b * N + i) * N + j] = v ? 1 : 0;
  }
}

}  // namespace spsattn
