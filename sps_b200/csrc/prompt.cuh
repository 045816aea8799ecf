// What a batched prompt prefill needs to know about its token ids, in one launch: the doubled ids
// and positions, the start of each row's document (what the attention's pre-pass would find out from
// document ids, once for all layers), which tokens belong to the last document, and the checks of the
// prompt.  Stands in for some 25 tensor operations and three host synchronisations.
// Reference: model.py:39-99 (left-padded checks, positions, document ids),
// reverse_sps/inference.py:615-660.
#pragma once

#include "common.cuh"

namespace spsattn {

struct PromptParams {
  const int64_t* ids;        // [B, T] contiguous
  int B, T, slots;
  int64_t eos, pad, predict;
  int empty_after_eos;       // a prompt that ends on EOS starts with empty caches (Standard model)
  int64_t* ids2;             // [B, T * slots]
  int64_t* pos2;             // [B, T * slots]
  int* run_start;            // [B, T * slots] first row of the row's document
  uint8_t* doc_mask;         // [B, T] token belongs to the last document
  int64_t* real_len;         // [B]
  uint8_t* ends_on_eos;      // [B]
  int64_t* flags;            // [4]: pad after a real token, row without a real token, longest row, status word; zeroed
  const int* status;
};

constexpr int kPromptThreads = 1024;

// One block per row.  A row's documents: every pad column is one of its own, then EOS tokens end them.
__global__ void __launch_bounds__(kPromptThreads) prompt_scan_kernel(const PromptParams p) {
  __shared__ int s_warp[3][kPromptThreads / 32];
  __shared__ int s_total[4];          // pads, EOS tokens before the last column, first real column, last pad column
  __shared__ int s_carry[3];
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t* ids = p.ids + (size_t)b * p.T;
  if (tid == 0) s_total[0] = s_total[1] = 0, s_total[2] = p.T, s_total[3] = -1, s_carry[0] = s_carry[1] = s_carry[2] = 0;
  __syncthreads();
  int pads = 0, eos = 0, first_real = p.T, last_pad = -1;
  for (int t = tid; t < p.T; t += kPromptThreads) {
    const int64_t id = ids[t];
    if (id == p.pad) {
      ++pads;
      last_pad = t;
    } else {
      first_real = min(first_real, t);
      if (id == p.eos && t < p.T - 1) ++eos;
    }
  }
  pads = __reduce_add_sync(0xffffffffu, pads);
  eos = __reduce_add_sync(0xffffffffu, eos);
  first_real = __reduce_min_sync(0xffffffffu, first_real);
  last_pad = __reduce_max_sync(0xffffffffu, last_pad);
  if (lane == 0) {
    atomicAdd(&s_total[0], pads);
    atomicAdd(&s_total[1], eos);
    atomicMin(&s_total[2], first_real);
    atomicMax(&s_total[3], last_pad);
  }
  __syncthreads();
  const int real = p.T - s_total[0], eos_total = s_total[1];
  const bool ends_on_eos = p.T > 0 && ids[p.T - 1] == p.eos;
  if (tid == 0) {
    p.real_len[b] = real;
    p.ends_on_eos[b] = ends_on_eos;
    if (s_total[3] > s_total[2]) p.flags[0] = 1;
    if (real == 0) p.flags[1] = 1;
    atomicMax(reinterpret_cast<unsigned long long*>(&p.flags[2]), (unsigned long long)real);
    if (b == 0 && p.status != nullptr) p.flags[3] = *p.status;
  }
  // running over the columns: real tokens, EOS tokens, latest start of a document
  for (int t0 = 0; t0 < p.T; t0 += kPromptThreads) {
    const int t = t0 + tid;
    const bool in = t < p.T;
    const int64_t id = in ? ids[t] : p.pad;
    const bool is_real = in && id != p.pad;
    const int64_t before = in && t > 0 ? ids[t - 1] : p.pad;
    // the first column, every pad, the first real token after pads, and what follows an EOS
    const bool start = in && (t == 0 || !is_real || before == p.pad || before == p.eos);
    int n_real = is_real, n_eos = is_real && t > 0 && before != p.pad && before == p.eos, from = start ? t : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int a = __shfl_up_sync(0xffffffffu, n_real, o), e = __shfl_up_sync(0xffffffffu, n_eos, o),
                f = __shfl_up_sync(0xffffffffu, from, o);
      if (lane >= o) {
        n_real += a;
        n_eos += e;
        from = max(from, f);
      }
    }
    if (lane == 31) s_warp[0][warp] = n_real, s_warp[1][warp] = n_eos, s_warp[2][warp] = from;
    __syncthreads();
    if (warp == 0) {
      int a = s_warp[0][lane], e = s_warp[1][lane], f = s_warp[2][lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int a2 = __shfl_up_sync(0xffffffffu, a, o), e2 = __shfl_up_sync(0xffffffffu, e, o),
                  f2 = __shfl_up_sync(0xffffffffu, f, o);
        if (lane >= o) a += a2, e += e2, f = max(f, f2);
      }
      s_warp[0][lane] = a, s_warp[1][lane] = e, s_warp[2][lane] = f;
    }
    __syncthreads();
    n_real += s_carry[0] + (warp > 0 ? s_warp[0][warp - 1] : 0);
    n_eos += s_carry[1] + (warp > 0 ? s_warp[1][warp - 1] : 0);
    from = max(from, max(s_carry[2], warp > 0 ? s_warp[2][warp - 1] : 0));
    if (in) {
      p.doc_mask[(size_t)b * p.T + t] = is_real && n_eos == eos_total && !(p.empty_after_eos && ends_on_eos);
      for (int s = 0; s < p.slots; ++s) {
        const size_t row = ((size_t)b * p.T + t) * p.slots + s;
        p.ids2[row] = s == 0 ? id : p.predict;
        p.pos2[row] = is_real ? n_real - 1 : 0;
        p.run_start[row] = from * p.slots;
      }
    }
    __syncthreads();
    if (tid == kPromptThreads - 1) s_carry[0] = n_real, s_carry[1] = n_eos, s_carry[2] = from;
    __syncthreads();
  }
}

}  // namespace spsattn
