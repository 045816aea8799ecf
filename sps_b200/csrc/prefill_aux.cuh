// Small kernels around the prefill path: the document pre-pass and the visibility test hook.
#pragma once

#include "common.cuh"
#include "mask.cuh"

namespace spsattn {

__device__ __forceinline__ long long load_doc(const void* docs, int is_i64, size_t off) {
  return is_i64 ? reinterpret_cast<const long long*>(docs)[off]
                : (long long)reinterpret_cast<const int*>(docs)[off];
}

// One block per batch row: lo[b][i] = first row of the run of equal ids containing row i, mono[b] = 1
// iff the ids never decrease.  Bound by latency (a few thousand ids): every warp asks for the ids of 256
// consecutive rows at once, coalesced, finds the run starts of 32 rows by a ballot, and one barrier
// carries the last start of each warp to those after it.  (With eight neighbouring rows per thread and a
// shuffle scan over them: 5.3 instead of 3.6 us at 3 x 3001 rows and 10.1 instead of 4.7 at 8 x 8192.)
__global__ void __launch_bounds__(1024)
doc_prepass_kernel(const void* docs, int is_i64, int64_t stride_b, int64_t stride_t, int N,
                   int* __restrict__ lo, int* __restrict__ mono, int* __restrict__ work_counter) {
  constexpr int kItems = 8;            // rows up to 8192 need a single pass
  __shared__ int s_last[2][32];        // last run start of a warp's rows (two passes' worth)
  const int b = blockIdx.x;
  const int tid = threadIdx.x;
  const int lane = tid & 31, warp = tid >> 5;
  // the attention kernel behind this one may be launched as a programmatic dependent: let its
  // blocks take the free SMs now (it waits for this grid before it reads lo / mono)
  grid_launch_dependents();
  const uint8_t* base =
      reinterpret_cast<const uint8_t*>(docs) + (size_t)b * stride_b * (is_i64 ? 8 : 4);
  // the attention kernel that follows in the stream draws its work items from this counter
  if (tid == 0 && b == 0 && work_counter != nullptr) *work_counter = 0;
  int carry = 0, decreases = 0;
  for (int c0 = 0, pass = 0; c0 < N; c0 += 1024 * kItems, pass ^= 1) {
    const int w0 = c0 + warp * 32 * kItems;
    long long id[kItems], edge = 0;
#pragma unroll
    for (int x = 0; x < kItems; ++x) {
      const int i = w0 + x * 32 + lane;
      id[x] = i < N ? load_doc(base, is_i64, (size_t)i * stride_t) : 0;
    }
    if (lane == 0 && w0 > 0 && w0 < N) edge = load_doc(base, is_i64, (size_t)(w0 - 1) * stride_t);
    int start[kItems], last = 0;       // run starts as far as this warp's rows tell
    bool dec = false;
#pragma unroll
    for (int x = 0; x < kItems; ++x) {
      const int i = w0 + x * 32 + lane;
      long long prev = __shfl_up_sync(0xffffffffu, id[x], 1);
      const long long tail = x > 0 ? __shfl_sync(0xffffffffu, id[x > 0 ? x - 1 : 0], 31) : edge;
      if (lane == 0) prev = tail;
      const bool inside = i > 0 && i < N;
      dec |= inside && id[x] < prev;
      const uint32_t starts = __ballot_sync(0xffffffffu, inside && id[x] != prev);
      const uint32_t upto = starts & (0xffffffffu >> (31 - lane));
      start[x] = upto ? i - lane + 31 - __clz(upto) : last;
      if (starts) last = w0 + x * 32 + 31 - __clz(starts);
    }
    if (lane == 0) s_last[pass][warp] = last;
    decreases |= __syncthreads_or(dec);
    const int of_warp = s_last[pass][lane];
    const int before = max(carry, __reduce_max_sync(0xffffffffu, lane < warp ? of_warp : 0));
    carry = max(carry, __reduce_max_sync(0xffffffffu, of_warp));
#pragma unroll
    for (int x = 0; x < kItems; ++x) {
      const int i = w0 + x * 32 + lane;
      if (i < N) lo[(size_t)b * N + i] = max(start[x], before);
    }
  }
  if (tid == 0) mono[b] = decreases ? 0 : 1;
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
