// Segmented decode attention: nq (1 or 2) queries per (sequence, head) over up to three
// length-masked KV segments plus up to two single-token "current" entries.
//
// The job is bandwidth bound (every live K/V row is read exactly once, both queries share the
// load), so it is split-K: the live rows of one (sequence, head) — the segments laid end to
// end — are cut into chunks of `chunk_rows`, one block per chunk.  A block streams its rows with
// 128-bit loads (D/8 lanes per row, four row batches in flight per lane), keeps an online
// softmax per lane group in fp32, merges the groups and writes one (max, sum, acc[D]) record
// per query into the workspace; a second small kernel merges the records of each
// (sequence, head) and writes the output (fp32, or 16-bit for a caller that feeds a projection).
// Lengths are read on the device, so the grid is sized from the host-side caps and blocks past
// the live length return at once.
// The decode-step form is a single launch: every block of a (sequence, head) takes a ticket when
// it is done and the last one merges the records itself, and (when asked) also performs the step's
// cache update for its (sequence, head) — ring insert, retained append, counters.  By then every
// block of that (sequence, head) has read the counters and finished reading the rows, which is
// what makes the in-place update safe; the per-sequence ring counters are advanced by the last
// (sequence, head) of the sequence to finish, through a second ticket.  Nothing waits on a ticket.
// Reference computation: src/modeling/models/utils/decode_attention.py:191-368 and, for the
// update, src/modeling/models/utils/decode_attention_fast.py:34-136.
#pragma once

#include "common.cuh"

namespace spsattn {

constexpr int kMaxSegments = 3;
constexpr int kMaxExtras = 2;
constexpr int kDecodeThreads = 128;
constexpr int kDecodeUnroll = 4;

struct DecodeSeg {
  const void* k;
  const void* v;
  const int64_t* seq_offset;
  int64_t seq_stride, head_stride, row_stride;
  const int64_t* lengths;
  int lengths_per_head;
  int max_rows;
  uint32_t query_mask;
};

// The cache update folded into the merge kernel (all pointers null = no update).
struct DecodeAppend {
  uint16_t* nw_k;            // ring      [S, H, window_storage, D]
  uint16_t* nw_v;
  int64_t* nw_len;           // [S]
  int64_t* nw_pos;           // [S]
  uint16_t* br_k;            // retained  [S, H, retained_storage, D]
  uint16_t* br_v;
  int64_t* br_len;           // [S, H]
  const uint16_t* k_window;  // [S, H, D]
  const uint16_t* v_window;
  const uint16_t* k_retained;
  const uint16_t* v_retained;
  const int8_t* active;      // [S]
  int window_storage, retained_storage, window_tokens;
  int ring_later;            // decode_pair_kernel: a later launch advances the ring counters
};

struct DecodeParams {
  const void* q;       // [S, nq, H, D]
  void* out;           // [S, nq, H, D] fp32, or 16-bit in the queries' format when out16 is set
  int out16;
  float* partial;      // [S*H][n_chunks][nq][D + 2]
  int* tickets;        // [S*H + S] zero before the first launch, left zero; null = separate merge launch
  // Tensor-core kernel only: records are indexed by slot = (segment, chunk inside the segment),
  // segment after segment, then one slot for the current-token entries.
  int seg_chunks[kMaxSegments];   // 0 for the short segments of small_segs
  int extras_slot;     // slot of the current-token entries and the short segments, -1 when none
  int pair;            // one block per (sequence, head): decode_pair_kernel
  int early_rows;      // decode_pair_kernel: nothing launched just before writes the segments' rows
  uint32_t small_segs; // bit x: segment x is short and handled with the entries, on the CUDA cores
  int* status;         // bounded-wait failures are reported here (may be null)
  DecodeAppend app;
  DecodeSeg seg[kMaxSegments];
  const void* extra_k[kMaxExtras];
  const void* extra_v[kMaxExtras];
  uint32_t extra_mask[kMaxExtras];
  int n_segments, n_extras;
  int S, H, nq;
  int chunk_rows, n_chunks;
  float scale_log2;
};

__device__ __forceinline__ int live_rows(const DecodeSeg& sg, int s, int h, int H) {
  long long len = sg.lengths_per_head ? sg.lengths[(size_t)s * H + h] : sg.lengths[s];
  if (len < 0) len = 0;
  return len < sg.max_rows ? (int)len : sg.max_rows;
}

// Merge the chunk records of one (sequence, head) and write its outputs; `nthreads` threads of
// one block cooperate.  Records are read past L1 (other blocks may have written them), eight
// chunks at a time with all their loads in flight together, so a merge costs about one round
// trip to L2 instead of one per chunk.
template <int D, int NQ, bool FP16>
__device__ __forceinline__ void merge_records(const DecodeParams& prm, int sh, int s, int h, int n_total,
                                              int tid, int nthreads) {
  constexpr int G = 8;
  int n_chunks = (n_total + prm.chunk_rows - 1) / prm.chunk_rows;
  if (n_chunks < 1) n_chunks = 1;
  for (int idx = tid; idx < NQ * D; idx += nthreads) {
    const int qi = idx / D, d = idx % D;
    const float* rec0 = prm.partial + (size_t)sh * prm.n_chunks * NQ * (D + 2) + qi * (D + 2);
    float m_run = -1.0e30f, l_run = 0.f, a_run = 0.f;
    for (int c0 = 0; c0 < n_chunks; c0 += G) {
      float m[G], l[G], a[G];
#pragma unroll
      for (int j = 0; j < G; ++j) {
        const int c = min(c0 + j, n_chunks - 1);      // clamped: the tail repeats a valid record
        const float* rec = rec0 + (size_t)c * NQ * (D + 2);
        m[j] = __ldcg(rec);
        l[j] = __ldcg(rec + 1);
        a[j] = __ldcg(rec + 2 + d);
      }
      float mx = m_run;
#pragma unroll
      for (int j = 0; j < G; ++j) mx = fmaxf(mx, m[j]);
      const float keep = fast_exp2(m_run - mx);
      l_run *= keep;
      a_run *= keep;
#pragma unroll
      for (int j = 0; j < G; ++j) {
        const float f = c0 + j < n_chunks ? fast_exp2(m[j] - mx) : 0.f;
        l_run = fmaf(l[j], f, l_run);
        a_run = fmaf(a[j], f, a_run);
      }
      m_run = mx;
    }
    const float o = l_run > 0.f ? a_run / l_run : 0.f;
    const size_t off = (((size_t)s * NQ + qi) * prm.H + h) * D + d;
    if (prm.out16)
      reinterpret_cast<uint16_t*>(prm.out)[off] = (uint16_t)(pack2<FP16>(o, 0.f) & 0xffffu);
    else
      reinterpret_cast<float*>(prm.out)[off] = o;
  }
}

// The same merge for the slot layout of the tensor-core kernel: a slot holds a record iff its
// chunk starts below the live length of its segment (the slot of the current-token entries and
// the short segments always does).  `seg_live[x]` = live rows of segment x.
template <int D, int NQ, bool FP16>
__device__ __forceinline__ void merge_slots(const DecodeParams& prm, int sh, int s, int h,
                                            const int (&seg_live)[kMaxSegments], int tid, int nthreads) {
  constexpr int G = 8;
  const int n_slots = prm.n_chunks;
  for (int idx = tid; idx < NQ * D; idx += nthreads) {
    const int qi = idx / D, d = idx % D;
    const float* rec0 = prm.partial + (size_t)sh * prm.n_chunks * NQ * (D + 2) + qi * (D + 2);
    float m_run = -1.0e30f, l_run = 0.f, a_run = 0.f;
    for (int c0 = 0; c0 < n_slots; c0 += G) {
      float m[G], l[G], a[G];
#pragma unroll
      for (int j = 0; j < G; ++j) {
        const int c = c0 + j;
        bool live = false;
        if (c < n_slots) {
          if (c == prm.extras_slot) {
            live = true;
          } else {
            int cc = c;
#pragma unroll
            for (int x = 0; x < kMaxSegments; ++x) {
              if (cc >= 0 && cc < prm.seg_chunks[x]) live = cc * prm.chunk_rows < seg_live[x];
              cc -= prm.seg_chunks[x];
            }
          }
        }
        const float* rec = rec0 + (size_t)(live ? c : 0) * NQ * (D + 2);
        m[j] = live ? __ldcg(rec) : -1.0e30f;
        l[j] = live ? __ldcg(rec + 1) : 0.f;
        a[j] = live ? __ldcg(rec + 2 + d) : 0.f;
      }
      float mx = m_run;
#pragma unroll
      for (int j = 0; j < G; ++j) mx = fmaxf(mx, m[j]);
      const float keep = fast_exp2(m_run - mx);
      l_run *= keep;
      a_run *= keep;
#pragma unroll
      for (int j = 0; j < G; ++j) {
        const float f = fast_exp2(m[j] - mx);
        l_run = fmaf(l[j], f, l_run);
        a_run = fmaf(a[j], f, a_run);
      }
      m_run = mx;
    }
    const float o = l_run > 0.f ? a_run / l_run : 0.f;
    const size_t off = (((size_t)s * NQ + qi) * prm.H + h) * D + d;
    if (prm.out16)
      reinterpret_cast<uint16_t*>(prm.out)[off] = (uint16_t)(pack2<FP16>(o, 0.f) & 0xffffu);
    else
      reinterpret_cast<float*>(prm.out)[off] = o;
  }
}

// End of a block of a single-launch decode: take the ticket of this (sequence, head); the last
// block to arrive merges the records, writes the output and applies the cache update.  Every
// block takes a ticket, also those past the live length, so that all of them have read the
// counters before any update.  `wrote` = this block stored a record (its stores are fenced).
// `local` (tensor-core kernel, one block per (sequence, head)): the block's two records — its
// tiles and the short segments / current entries — are in shared memory at `local`; there is
// nobody to take a ticket against, and the merge needs no trip through global memory.
template <int D, int NQ, bool FP16, bool SLOTS>
__device__ __forceinline__ void decode_finish(const DecodeParams& prm, int sh, int s, int h, int n_total,
                                              const int (&seg_live)[kMaxSegments], long long ring_len,
                                              long long ring_pos, long long ret_len, bool wrote, int tid,
                                              int nthreads, const float* local = nullptr,
                                              uint32_t local_live = 0) {
  if (local != nullptr) {
    __syncthreads();
    for (int idx = tid; idx < NQ * D; idx += nthreads) {
      const int qi = idx / D, d = idx % D;
      float m[2], l[2], a[2];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        const float* rec = local + (c * NQ + qi) * (D + 2);
        const bool live = (local_live >> c) & 1u;
        m[c] = live ? rec[0] : -1.0e30f;
        l[c] = live ? rec[1] : 0.f;
        a[c] = live ? rec[2 + d] : 0.f;
      }
      const float mx = fmaxf(m[0], m[1]);
      const float f0 = fast_exp2(m[0] - mx), f1 = fast_exp2(m[1] - mx);
      const float lsum = l[0] * f0 + l[1] * f1, asum = a[0] * f0 + a[1] * f1;
      const float o = lsum > 0.f ? asum / lsum : 0.f;
      const size_t off = (((size_t)s * NQ + qi) * prm.H + h) * D + d;
      if (prm.out16)
        reinterpret_cast<uint16_t*>(prm.out)[off] = (uint16_t)(pack2<FP16>(o, 0.f) & 0xffffu);
      else
        reinterpret_cast<float*>(prm.out)[off] = o;
    }
  } else {
    // (the barrier orders the block's record stores before thread 0's fence, which is cumulative)
    if (wrote) __syncthreads();
    __shared__ int s_last;
    if (tid == 0) {
      if (wrote) __threadfence();
      const bool last = atomicAdd(&prm.tickets[sh], 1) == (int)gridDim.y - 1;
      if (last) __threadfence();
      s_last = last;
    }
    __syncthreads();
    if (!s_last) return;
    if constexpr (SLOTS)
      merge_slots<D, NQ, FP16>(prm, sh, s, h, seg_live, tid, nthreads);
    else
      merge_records<D, NQ, FP16>(prm, sh, s, h, n_total, tid, nthreads);
  }
  const DecodeAppend& ap = prm.app;
  const bool append = ap.br_k != nullptr && ap.active[s] != 0;
  const bool full = ring_len >= ap.window_tokens;
  if (append) {
    const long long ins = full ? ring_pos : ring_len;
    for (int d = tid; d < D; d += nthreads) {
      const size_t src = (size_t)sh * D + d;
      if (ap.window_tokens > 0 && ins >= 0 && ins < ap.window_storage) {
        const size_t dst = ((size_t)sh * ap.window_storage + (size_t)ins) * D + d;
        ap.nw_k[dst] = ap.k_window[src];
        ap.nw_v[dst] = ap.v_window[src];
      }
      if (ret_len >= 0 && ret_len < ap.retained_storage) {
        const size_t dst = ((size_t)sh * ap.retained_storage + (size_t)ret_len) * D + d;
        ap.br_k[dst] = ap.k_retained[src];
        ap.br_v[dst] = ap.v_retained[src];
      }
    }
  }
  if (tid == 0) {
    if (local == nullptr) prm.tickets[sh] = 0;   // ready for the next launch
    if (append && ret_len < ap.retained_storage) ap.br_len[sh] = ret_len + 1;
    if (ap.br_k != nullptr && ap.window_tokens > 0) {
      // the ring counters belong to the sequence: the last of its heads to get here advances them
      __threadfence();
      int* seq_ticket = prm.tickets + (size_t)prm.S * prm.H + s;
      if (atomicAdd(seq_ticket, 1) == prm.H - 1) {
        *seq_ticket = 0;
        if (append) {
          if (full)
            ap.nw_pos[s] = (ring_pos + 1) % ap.window_tokens;
          else
            ap.nw_len[s] = ring_len + 1;
        }
      }
    }
  }
}

// The CUDA-core pass over rows [c_lo, c_hi) of the segments laid end to end (`seg_start` =
// running sum of their live rows), plus the current-token entries when asked, ending in one
// record per query at `rec`.  Run by the first kDecodeThreads threads of the block, all of which
// must call it (it synchronises them on named barrier 2; the other threads stay out).
template <int D, int NQ, bool FP16>
__device__ __forceinline__ void cuda_core_chunk(const DecodeParams& prm, int s, int h, int sh,
                                                const int (&seg_start)[kMaxSegments + 1], int c_lo, int c_hi,
                                                bool with_extras, float* rec, int tid) {
  constexpr int LPR = D / 8;          // lanes per row
  constexpr int RPI = 32 / LPR;       // rows per warp load instruction
  constexpr int U = kDecodeUnroll;
  constexpr int STEP = 4 * RPI * U;   // rows per block step
  static_assert(D % 8 == 0 && 32 % LPR == 0, "head_dim");
  const int warp = (tid >> 5) & 3, lane = tid & 31;
  const int g = lane / LPR;           // row inside a load instruction
  const int dl = (lane % LPR) * 8;    // first of this lane's 8 dims
  const bool worker = tid < kDecodeThreads;
  __shared__ float s_m[4][NQ], s_l[4][NQ], s_acc[4][NQ][D];
  if (worker) {
    if (with_extras && warp == 0 && lane < 2 * prm.n_extras) {
      // the single-row entries are read last, by one warp: have them in L2 by then
      const void* base = (lane & 1) ? prm.extra_v[lane >> 1] : prm.extra_k[lane >> 1];
      asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint16_t*>(base) + (size_t)sh * D));
    }
    // queries, pre-scaled so scores are in the log2 domain
    float q[NQ][8];
#pragma unroll
    for (int qi = 0; qi < NQ; ++qi) {
      const uint4 u = *reinterpret_cast<const uint4*>(
          reinterpret_cast<const uint16_t*>(prm.q) + (((size_t)s * NQ + qi) * prm.H + h) * D + dl);
      unpack2<FP16>(u.x, q[qi][0], q[qi][1]);
      unpack2<FP16>(u.y, q[qi][2], q[qi][3]);
      unpack2<FP16>(u.z, q[qi][4], q[qi][5]);
      unpack2<FP16>(u.w, q[qi][6], q[qi][7]);
#pragma unroll
      for (int x = 0; x < 8; ++x) q[qi][x] *= prm.scale_log2;
    }

    float m_run[NQ], l_run[NQ], acc[NQ][8];
#pragma unroll
    for (int qi = 0; qi < NQ; ++qi) {
      m_run[qi] = -1.0e30f;
      l_run[qi] = 0.f;
#pragma unroll
      for (int x = 0; x < 8; ++x) acc[qi][x] = 0.f;
    }

    // one batch of U rows (one per unroll slot) for this lane group
    auto process = [&](const uint16_t* kb, const uint16_t* vb, int64_t row_stride, int r0, int r_hi,
                       uint32_t qmask) {
      uint4 kr[U], vr[U];
      bool valid[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int r = r0 + u * (4 * RPI);
        valid[u] = r < r_hi;
        if (valid[u]) {
          kr[u] = __ldg(reinterpret_cast<const uint4*>(kb + (size_t)r * row_stride + dl));
          vr[u] = __ldg(reinterpret_cast<const uint4*>(vb + (size_t)r * row_stride + dl));
        } else {
          kr[u] = make_uint4(0, 0, 0, 0);
          vr[u] = make_uint4(0, 0, 0, 0);
        }
      }
      float sc[NQ][U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float kf[8];
        unpack2<FP16>(kr[u].x, kf[0], kf[1]);
        unpack2<FP16>(kr[u].y, kf[2], kf[3]);
        unpack2<FP16>(kr[u].z, kf[4], kf[5]);
        unpack2<FP16>(kr[u].w, kf[6], kf[7]);
#pragma unroll
        for (int qi = 0; qi < NQ; ++qi) {
          float d = 0.f;
#pragma unroll
          for (int x = 0; x < 8; ++x) d = fmaf(q[qi][x], kf[x], d);
#pragma unroll
          for (int o = LPR / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
          sc[qi][u] = (valid[u] && ((qmask >> qi) & 1u)) ? d : -INFINITY;
        }
      }
      float pr[NQ][U], alpha[NQ];
#pragma unroll
      for (int qi = 0; qi < NQ; ++qi) {
        float mx = m_run[qi];
#pragma unroll
        for (int u = 0; u < U; ++u) mx = fmaxf(mx, sc[qi][u]);
        alpha[qi] = fast_exp2(m_run[qi] - mx);
        float sum = 0.f;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          pr[qi][u] = fast_exp2(sc[qi][u] - mx);
          sum += pr[qi][u];
        }
        l_run[qi] = l_run[qi] * alpha[qi] + sum;
        m_run[qi] = mx;
#pragma unroll
        for (int x = 0; x < 8; ++x) acc[qi][x] *= alpha[qi];
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float vf[8];
        unpack2<FP16>(vr[u].x, vf[0], vf[1]);
        unpack2<FP16>(vr[u].y, vf[2], vf[3]);
        unpack2<FP16>(vr[u].z, vf[4], vf[5]);
        unpack2<FP16>(vr[u].w, vf[6], vf[7]);
#pragma unroll
        for (int qi = 0; qi < NQ; ++qi)
#pragma unroll
          for (int x = 0; x < 8; ++x) acc[qi][x] = fmaf(pr[qi][u], vf[x], acc[qi][x]);
      }
    };

#pragma unroll
    for (int x = 0; x < kMaxSegments; ++x) {
      if (x >= prm.n_segments) break;
      const int lo = max(c_lo, seg_start[x]) - seg_start[x];
      const int hi = min(c_hi, seg_start[x + 1]) - seg_start[x];
      if (lo >= hi) continue;
      const DecodeSeg& sg = prm.seg[x];
      const int64_t base = (sg.seq_offset ? sg.seq_offset[s] : (int64_t)s * sg.seq_stride) +
                           (int64_t)h * sg.head_stride;
      const uint16_t* kb = reinterpret_cast<const uint16_t*>(sg.k) + base;
      const uint16_t* vb = reinterpret_cast<const uint16_t*>(sg.v) + base;
      for (int r = lo + warp * RPI + g; r - (warp * RPI + g) < hi; r += STEP)
        process(kb, vb, sg.row_stride, r, hi, sg.query_mask);
    }
    if (with_extras && warp == 0) {
      // the current-token entries: one row each, handled by lane group 0 of warp 0
      for (int e = 0; e < prm.n_extras; ++e) {
        const uint16_t* kb = reinterpret_cast<const uint16_t*>(prm.extra_k[e]) + (size_t)sh * D;
        const uint16_t* vb = reinterpret_cast<const uint16_t*>(prm.extra_v[e]) + (size_t)sh * D;
        process(kb, vb, 0, g, 1, prm.extra_mask[e]);
      }
    }

    // merge the lane groups of a warp, then the four warps, then write the record
#pragma unroll
    for (int qi = 0; qi < NQ; ++qi) {
#pragma unroll
      for (int o = LPR; o < 32; o <<= 1) {
        const float m_o = __shfl_xor_sync(0xffffffffu, m_run[qi], o);
        const float l_o = __shfl_xor_sync(0xffffffffu, l_run[qi], o);
        const float mx = fmaxf(m_run[qi], m_o);
        const float a = fast_exp2(m_run[qi] - mx), bsc = fast_exp2(m_o - mx);
        l_run[qi] = l_run[qi] * a + l_o * bsc;
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          const float acc_o = __shfl_xor_sync(0xffffffffu, acc[qi][x], o);
          acc[qi][x] = acc[qi][x] * a + acc_o * bsc;
        }
        m_run[qi] = mx;
      }
    }
    if (g == 0) {
#pragma unroll
      for (int qi = 0; qi < NQ; ++qi) {
        if (lane == 0) {
          s_m[warp][qi] = m_run[qi];
          s_l[warp][qi] = l_run[qi];
        }
#pragma unroll
        for (int x = 0; x < 8; ++x) s_acc[warp][qi][dl + x] = acc[qi][x];
      }
    }
  }
  if (worker) asm volatile("bar.sync 2, %0;" ::"n"(kDecodeThreads) : "memory");
  if (worker) {
    for (int idx = tid; idx < NQ * D; idx += kDecodeThreads) {
      const int qi = idx / D, d = idx % D;
      float mx = s_m[0][qi];
#pragma unroll
      for (int w = 1; w < 4; ++w) mx = fmaxf(mx, s_m[w][qi]);
      float a = 0.f, l = 0.f;
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        const float f = fast_exp2(s_m[w][qi] - mx);
        a += s_acc[w][qi][d] * f;
        l += s_l[w][qi] * f;
      }
      rec[qi * (D + 2) + 2 + d] = a;
      if (d == 0) {
        rec[qi * (D + 2)] = mx;
        rec[qi * (D + 2) + 1] = l;
      }
    }
  }
}

template <int D, int NQ, bool FP16>
__global__ void __launch_bounds__(kDecodeThreads, 5)
decode_split_kernel(const DecodeParams prm) {
  const int sh = blockIdx.x;
  const int s = sh / prm.H, h = sh % prm.H;
  // highest chunk first: blocks past the live length retire at once, at the start of the launch
  const int chunk = (int)gridDim.y - 1 - (int)blockIdx.y;
  const int tid = threadIdx.x;
  grid_launch_dependents();
  grid_dependency_wait();      // in a decode step: the queries and counters come from the launch before

  int seg_start[kMaxSegments + 1];
  seg_start[0] = 0;
#pragma unroll
  for (int x = 0; x < kMaxSegments; ++x)
    seg_start[x + 1] = seg_start[x] + (x < prm.n_segments ? live_rows(prm.seg[x], s, h, prm.H) : 0);
  const int n_total = seg_start[kMaxSegments];
  const int c_lo = chunk * prm.chunk_rows;
  const bool dead = chunk > 0 && c_lo >= n_total;
  if (dead && prm.tickets == nullptr) return;
  const int c_hi = min(c_lo + prm.chunk_rows, n_total);
  // the counters as they are before this step's update (any block may be the one that applies it)
  long long ring_len = 0, ring_pos = 0, ret_len = 0;
  if (prm.app.br_len != nullptr) {
    ret_len = prm.app.br_len[(size_t)s * prm.H + h];
    if (prm.app.window_tokens > 0) {
      ring_len = prm.app.nw_len[s];
      ring_pos = prm.app.nw_pos[s];
    }
  }

  if (!dead) {   // blocks past the live length only take their ticket below
    float* rec = prm.partial + ((size_t)sh * prm.n_chunks + chunk) * NQ * (D + 2);
    cuda_core_chunk<D, NQ, FP16>(prm, s, h, sh, seg_start, c_lo, c_hi, chunk == 0, rec, tid);
  }

  if (prm.tickets == nullptr) return;     // a separate launch merges
  int seg_live[kMaxSegments];
#pragma unroll
  for (int x = 0; x < kMaxSegments; ++x) seg_live[x] = seg_start[x + 1] - seg_start[x];
  decode_finish<D, NQ, FP16, false>(prm, sh, s, h, n_total, seg_live, ring_len, ring_pos, ret_len, !dead,
                                    tid, kDecodeThreads);
}

// ---------------------------------------------------------------------------------------------
// The same attention with one block per (sequence, head), for few pairs with short caches, where a
// launch is bound by latency: a pair's chunks are taken by groups of 128 threads of one block and
// merged in its shared memory, so no record goes through global memory and no ticket is waited for
// (about 3 us), every batch of rows is asked for while the one before it is worked on, and the first
// batch is in registers before the launch that produces the queries has ended.  Chunks, batches and
// sums are those of decode_split_kernel, so the results are the same bits.
constexpr int kPairMaxChunks = 8;
constexpr int kPairMaxGroups = 4;

template <int D, int NQ>
struct PairScratch {
  float m[4][NQ], l[4][NQ], acc[4][NQ][D];
};

// Live rows of the segments, laid end to end.  The lengths are asked for together: one at a time, each
// behind a branch, they and the counters were 3200 of the block's 11000 clocks.
struct PairLengths {
  long long raw[kMaxSegments];
  __device__ __forceinline__ void ask(const DecodeParams& prm, int s, int sh) {
#pragma unroll
    for (int x = 0; x < kMaxSegments; ++x) {
      const DecodeSeg& sg = prm.seg[x];
      raw[x] = 0;
      if (x < prm.n_segments) raw[x] = __ldcg(sg.lengths + (sg.lengths_per_head ? sh : s));
    }
  }
  __device__ __forceinline__ void starts(const DecodeParams& prm, int (&seg_start)[kMaxSegments + 1]) const {
    seg_start[0] = 0;
#pragma unroll
    for (int x = 0; x < kMaxSegments; ++x) {
      const long long len = raw[x] < 0 ? 0 : raw[x];
      seg_start[x + 1] = seg_start[x] + (x >= prm.n_segments ? 0 : len < prm.seg[x].max_rows ? (int)len : prm.seg[x].max_rows);
    }
  }
};

// A lane's batch of rows r, r + 4 RPI, ... (kDecodeUnroll of them) of segment x; the next one is
// 4 RPI kDecodeUnroll rows further on, or the first of a later segment.
struct PairBatch {
  int x, r, hi;
  int64_t row_stride;
  uint32_t mask;
  const uint16_t *kb, *vb;
};

// First batch of the chunk [c_lo, c_hi) in segment b.x or a later one; `off`: this lane's row in it.
__device__ __forceinline__ void pair_enter(const DecodeParams& prm, int s, int h, const int (&seg_start)[kMaxSegments + 1],
                                           int c_lo, int c_hi, int off, int dl, PairBatch& b) {
  const int from = b.x;
  b.x = kMaxSegments;
#pragma unroll
  for (int x = kMaxSegments - 1; x >= 0; --x) {
    const int lo = max(c_lo, seg_start[x]) - seg_start[x], hi = min(c_hi, seg_start[x + 1]) - seg_start[x];
    if (x < from || x >= prm.n_segments || lo >= hi) continue;
    const DecodeSeg& sg = prm.seg[x];
    const int64_t base = (sg.seq_offset ? sg.seq_offset[s] : (int64_t)s * sg.seq_stride) + (int64_t)h * sg.head_stride + dl;
    b.x = x;
    b.hi = hi;
    b.r = lo + off;
    b.row_stride = sg.row_stride;
    b.mask = sg.query_mask;
    b.kb = reinterpret_cast<const uint16_t*>(sg.k) + base;
    b.vb = reinterpret_cast<const uint16_t*>(sg.v) + base;
  }
}

template <int RPI>
__device__ __forceinline__ void pair_load(const uint16_t* base, const PairBatch& b, uint4 (&rows)[kDecodeUnroll]) {
#pragma unroll
  for (int u = 0; u < kDecodeUnroll; ++u) {
    const int r = b.r + u * (4 * RPI);
    rows[u] = make_uint4(0, 0, 0, 0);
    if (r < b.hi) rows[u] = __ldg(reinterpret_cast<const uint4*>(base + (size_t)r * b.row_stride));
  }
}

// `cur`, kr, vr: the chunk's first batch and its rows; `entries`: current-token rows in shared memory, K
// and V in turn, copied there by the warp that reads them (asynchronously, it still has to wait)
template <int D, int NQ, bool FP16>
__device__ __forceinline__ void pair_chunk(const DecodeParams& prm, int s, int h, int sh,
                                           const int (&seg_start)[kMaxSegments + 1], int c_lo, int c_hi,
                                           bool with_extras, float* rec, int tid, PairScratch<D, NQ>& scratch, int bar_id,
                                           const uint4 (&q_raw)[NQ], uint32_t entries, PairBatch cur, uint4 (&kr)[kDecodeUnroll],
                                           uint4 (&vr)[kDecodeUnroll]) {
  constexpr int LPR = D / 8;          // lanes per row
  constexpr int RPI = 32 / LPR;       // rows per warp load instruction
  constexpr int U = kDecodeUnroll;
  constexpr int STEP = 4 * RPI * U;   // rows per step of the group
  const int warp = tid >> 5, lane = tid & 31;
  const int g = lane / LPR;           // row inside a load instruction
  const int dl = (lane % LPR) * 8;    // first of this lane's 8 dims
  const int off = warp * RPI + g;
  const bool extras = with_extras && warp == 0;
  float q[NQ][8], m_run[NQ], l_run[NQ], acc[NQ][8];
#pragma unroll
  for (int qi = 0; qi < NQ; ++qi) {
    m_run[qi] = -1.0e30f;
    l_run[qi] = 0.f;
#pragma unroll
    for (int x = 0; x < 8; ++x) acc[qi][x] = 0.f;
  }
  auto unpack8 = [](const uint4& u, float (&f)[8]) {
    unpack2<FP16>(u.x, f[0], f[1]);
    unpack2<FP16>(u.y, f[2], f[3]);
    unpack2<FP16>(u.z, f[4], f[5]);
    unpack2<FP16>(u.w, f[6], f[7]);
  };
  // `ahead` runs between the scores and the sums: the keys are done with there
  auto compute = [&](const uint4 (&kr)[U], const uint4 (&vr)[U], int r0, int r_hi, uint32_t qmask, auto ahead) {
    float sc[NQ][U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float kf[8];
      unpack8(kr[u], kf);
#pragma unroll
      for (int qi = 0; qi < NQ; ++qi) {
        float d = 0.f;
#pragma unroll
        for (int x = 0; x < 8; ++x) d = fmaf(q[qi][x], kf[x], d);
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        sc[qi][u] = (r0 + u * (4 * RPI) < r_hi && ((qmask >> qi) & 1u)) ? d : -INFINITY;
      }
    }
    ahead();
    float pr[NQ][U];
#pragma unroll
    for (int qi = 0; qi < NQ; ++qi) {
      float mx = m_run[qi];
#pragma unroll
      for (int u = 0; u < U; ++u) mx = fmaxf(mx, sc[qi][u]);
      const float alpha = fast_exp2(m_run[qi] - mx);
      float sum = 0.f;
#pragma unroll
      for (int u = 0; u < U; ++u) {
        pr[qi][u] = fast_exp2(sc[qi][u] - mx);
        sum += pr[qi][u];
      }
      l_run[qi] = l_run[qi] * alpha + sum;
      m_run[qi] = mx;
#pragma unroll
      for (int x = 0; x < 8; ++x) acc[qi][x] *= alpha;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float vf[8];
      unpack8(vr[u], vf);
#pragma unroll
      for (int qi = 0; qi < NQ; ++qi)
#pragma unroll
        for (int x = 0; x < 8; ++x) acc[qi][x] = fmaf(pr[qi][u], vf[x], acc[qi][x]);
    }
  };

#pragma unroll
  for (int qi = 0; qi < NQ; ++qi) {
    // pre-scaled so that scores are in the log2 domain
    unpack8(q_raw[qi], q[qi]);
#pragma unroll
    for (int x = 0; x < 8; ++x) q[qi][x] *= prm.scale_log2;
  }
  while (cur.x < kMaxSegments) {
    PairBatch next = cur;
    next.r += STEP;
    if (next.r - off >= next.hi) {
      ++next.x;
      pair_enter(prm, s, h, seg_start, c_lo, c_hi, off, dl, next);
    }
    const bool more = next.x < kMaxSegments;
    compute(kr, vr, cur.r, cur.hi, cur.mask, [&]() {
      if (more) pair_load<RPI>(next.kb, next, kr);
    });
    if (more) pair_load<RPI>(next.vb, next, vr);
    cur = next;
  }
  if (extras) {
    // one row each, in lane group 0, one after the other; their scores are made at once
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
    float sc[kMaxExtras][NQ];
#pragma unroll
    for (int e = 0; e < kMaxExtras; ++e) {
      if (e >= prm.n_extras) break;
      float kf[8];
      unpack8(lds16(entries + (2 * e * D + dl) * 2), kf);
#pragma unroll
      for (int qi = 0; qi < NQ; ++qi) {
        float d = 0.f;
#pragma unroll
        for (int x = 0; x < 8; ++x) d = fmaf(q[qi][x], kf[x], d);
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        sc[e][qi] = g == 0 && ((prm.extra_mask[e] >> qi) & 1u) ? d : -INFINITY;
      }
    }
#pragma unroll
    for (int e = 0; e < kMaxExtras; ++e) {
      if (e >= prm.n_extras) break;
      float vf[8];
      unpack8(lds16(entries + ((2 * e + 1) * D + dl) * 2), vf);
#pragma unroll
      for (int qi = 0; qi < NQ; ++qi) {
        const float mx = fmaxf(m_run[qi], sc[e][qi]);
        const float alpha = fast_exp2(m_run[qi] - mx), p = fast_exp2(sc[e][qi] - mx);
        l_run[qi] = l_run[qi] * alpha + p;
        m_run[qi] = mx;
#pragma unroll
        for (int x = 0; x < 8; ++x) acc[qi][x] = fmaf(p, vf[x], acc[qi][x] * alpha);
      }
    }
  }

  // merge the lane groups of a warp, then the four warps, then write the record
#pragma unroll
  for (int qi = 0; qi < NQ; ++qi) {
#pragma unroll
    for (int o = LPR; o < 32; o <<= 1) {
      const float m_o = __shfl_xor_sync(0xffffffffu, m_run[qi], o);
      const float l_o = __shfl_xor_sync(0xffffffffu, l_run[qi], o);
      const float mx = fmaxf(m_run[qi], m_o);
      const float a = fast_exp2(m_run[qi] - mx), bsc = fast_exp2(m_o - mx);
      l_run[qi] = l_run[qi] * a + l_o * bsc;
#pragma unroll
      for (int x = 0; x < 8; ++x) {
        const float acc_o = __shfl_xor_sync(0xffffffffu, acc[qi][x], o);
        acc[qi][x] = acc[qi][x] * a + acc_o * bsc;
      }
      m_run[qi] = mx;
    }
    if (g == 0) {
      if (lane == 0) {
        scratch.m[warp][qi] = m_run[qi];
        scratch.l[warp][qi] = l_run[qi];
      }
#pragma unroll
      for (int x = 0; x < 8; ++x) scratch.acc[warp][qi][dl + x] = acc[qi][x];
    }
  }
  asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "n"(kDecodeThreads) : "memory");
  for (int idx = tid; idx < NQ * D; idx += kDecodeThreads) {
    const int qi = idx / D, d = idx % D;
    float mx = scratch.m[0][qi];
#pragma unroll
    for (int v = 1; v < 4; ++v) mx = fmaxf(mx, scratch.m[v][qi]);
    float a = 0.f, l = 0.f;
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const float f = fast_exp2(scratch.m[v][qi] - mx);
      a += scratch.acc[v][qi][d] * f;
      l += scratch.l[v][qi] * f;
    }
    rec[qi * (D + 2) + 2 + d] = a;
    if (d == 0) {
      rec[qi * (D + 2)] = mx;
      rec[qi * (D + 2) + 1] = l;
    }
  }
}

template <int D, int NQ, bool FP16>
__global__ void __launch_bounds__(kPairMaxGroups * kDecodeThreads, 1) decode_pair_kernel(const DecodeParams prm) {
  __shared__ PairScratch<D, NQ> s_scratch[kPairMaxGroups];
  __shared__ float s_record[kPairMaxChunks][NQ * (D + 2)];
  __shared__ __align__(16) uint16_t s_rows[(2 * kMaxExtras + 4) * D];     // current-token entries, rows to store
  const int sh = blockIdx.x;
  const int s = sh / prm.H, h = sh % prm.H;
  const int tid = threadIdx.x, group = tid / kDecodeThreads, gt = tid % kDecodeThreads;
  const int groups = blockDim.x / kDecodeThreads;
  grid_launch_dependents();
  const DecodeAppend& ap = prm.app;
  constexpr int RPI = 32 / (D / 8);
  const int lane = gt & 31, off = (gt >> 5) * RPI + lane / (D / 8), dl = (lane % (D / 8)) * 8;
  auto first_batch = [&](const int (&seg_start)[kMaxSegments + 1], int c, PairBatch& cur, uint4 (&kr)[kDecodeUnroll],
                         uint4 (&vr)[kDecodeUnroll]) {
    cur.x = 0;
    pair_enter(prm, s, h, seg_start, c * prm.chunk_rows, min((c + 1) * prm.chunk_rows, seg_start[kMaxSegments]), off, dl, cur);
    if (cur.x < kMaxSegments) {
      pair_load<RPI>(cur.kb, cur, kr);
      pair_load<RPI>(cur.vb, cur, vr);
    }
  };
  // Inside a decode step of a decoder nothing from its start on writes these rows (the launch that
  // starts the step lets its dependents go only when everything before it is complete), so the first
  // batch may be read and the other rows sent for before the wait.  Only the lengths may still be about
  // to be reset: they are looked at again.
  int seg_start[kMaxSegments + 1] = {};
  PairBatch cur;
  uint4 kr[kDecodeUnroll], vr[kDecodeUnroll];
  bool same = prm.early_rows != 0;
  if (same) {
    PairLengths lengths;
    lengths.ask(prm, s, sh);
    lengths.starts(prm, seg_start);
    first_batch(seg_start, group, cur, kr, vr);
  }
#pragma unroll
  for (int x = 0; x < kMaxSegments; ++x) {
    if (x >= prm.n_segments || !same) break;
    const DecodeSeg& sg = prm.seg[x];
    if (sg.seq_offset != nullptr) continue;
    const int live = seg_start[x + 1] - seg_start[x];
    const int64_t base = (int64_t)s * sg.seq_stride + (int64_t)h * sg.head_stride;
    for (int r = tid; r < live; r += blockDim.x) {
#pragma unroll
      for (int e = 0; e < D; e += 64) {        // lines of 128 bytes
        asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint16_t*>(sg.k) + base + r * sg.row_stride + e));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint16_t*>(sg.v) + base + r * sg.row_stride + e));
      }
    }
  }
  grid_dependency_wait();

  // What the block needs from memory now is asked for at once: the queries and current-token entries, the
  // lengths, the counters as they are before this step's update, and (a thread each) the vectors of the
  // new rows: K and V for the retained cache, K and V for the ring.
  uint4 q_raw[NQ];
  PairLengths lengths;
#pragma unroll
  for (int qi = 0; qi < NQ; ++qi)
    q_raw[qi] = __ldcg(reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(prm.q) +
                                                      (((size_t)s * NQ + qi) * prm.H + h) * D + dl));
  lengths.ask(prm, s, sh);
  constexpr int kRowVecs = D / 8;
  const uint32_t entries = smem_u32(s_rows), new_rows = entries + 2 * kMaxExtras * D * 2;
  if (tid < 32)
    for (int i = tid; i < 2 * prm.n_extras * kRowVecs; i += 32) {
      const int row = i / kRowVecs;
      const void* src = (row & 1) ? prm.extra_v[row >> 1] : prm.extra_k[row >> 1];
      copy16(entries + i * 16, reinterpret_cast<const uint16_t*>(src) + (size_t)sh * D + (i - row * kRowVecs) * 8);
    }
  long long ring_len = 0, ring_pos = 0, ret_len = 0;
  int8_t active = 0;
  const int kind = tid / kRowVecs;
  if (ap.br_len != nullptr) {
    active = __ldcg(ap.active + s);
    ret_len = __ldcg(ap.br_len + sh);
    if (ap.window_tokens > 0) {
      ring_len = __ldcg(ap.nw_len + s);
      ring_pos = __ldcg(ap.nw_pos + s);
    }
    if (kind < (ap.window_tokens > 0 ? 4 : 2)) {
      const uint16_t* src = kind == 0 ? ap.k_retained : kind == 1 ? ap.v_retained : kind == 2 ? ap.k_window : ap.v_window;
      copy16(new_rows + tid * 16, src + (size_t)sh * D + tid % kRowVecs * 8);
    }
  }
  {
    int now[kMaxSegments + 1];
    lengths.starts(prm, now);
#pragma unroll
    for (int x = 1; x <= kMaxSegments; ++x) {
      same = same && now[x] == seg_start[x];
      seg_start[x] = now[x];
    }
    if (!same) first_batch(seg_start, group, cur, kr, vr);
  }
  const int n_total = seg_start[kMaxSegments];
  const int chunks = max(1, (n_total + prm.chunk_rows - 1) / prm.chunk_rows);
  for (int c = group; c < chunks; c += groups) {
    // (the record of the group's chunk before is complete: its scratch may be written again)
    if (c >= groups) {
      first_batch(seg_start, c, cur, kr, vr);
      asm volatile("bar.sync %0, %1;" ::"r"(2 + group), "n"(kDecodeThreads) : "memory");
    }
    pair_chunk<D, NQ, FP16>(prm, s, h, sh, seg_start, c * prm.chunk_rows, min((c + 1) * prm.chunk_rows, n_total), c == 0,
                            s_record[c], gt, s_scratch[group], 2 + group, q_raw, entries, cur, kr, vr);
  }
  __syncthreads();
  // merge_records on shared memory: one group of eight
  for (int idx = tid; idx < NQ * D; idx += blockDim.x) {
    const int qi = idx / D, d = idx % D;
    float mx = -1.0e30f;
    for (int j = 0; j < chunks; ++j) mx = fmaxf(mx, s_record[j][qi * (D + 2)]);
    float l_run = 0.f, a_run = 0.f;
    for (int j = 0; j < chunks; ++j) {
      const float* rec = s_record[j] + qi * (D + 2);
      const float f = fast_exp2(rec[0] - mx);
      l_run = fmaf(rec[1], f, l_run);
      a_run = fmaf(rec[2 + d], f, a_run);
    }
    const float o = l_run > 0.f ? a_run / l_run : 0.f;
    const size_t at = (((size_t)s * NQ + qi) * prm.H + h) * D + d;
    if (prm.out16)
      reinterpret_cast<uint16_t*>(prm.out)[at] = (uint16_t)(pack2<FP16>(o, 0.f) & 0xffffu);
    else
      reinterpret_cast<float*>(prm.out)[at] = o;
  }
  if (ap.br_k == nullptr) return;
  // the pair's rows have all been read: its new rows may be stored
  asm volatile("cp.async.wait_all;" ::: "memory");
  const bool full = ring_len >= ap.window_tokens, append = active != 0;
  if (append && kind < 4) {
    const bool ring = kind >= 2;
    const long long at = ring ? (full ? ring_pos : ring_len) : ret_len;
    const int storage = ring ? ap.window_storage : ap.retained_storage;
    uint16_t* dst = kind == 0 ? ap.br_k : kind == 1 ? ap.br_v : kind == 2 ? ap.nw_k : ap.nw_v;
    if ((!ring || ap.window_tokens > 0) && at >= 0 && at < storage)
      reinterpret_cast<uint4*>(dst + ((size_t)sh * storage + (size_t)at) * D)[tid % kRowVecs] = lds16(new_rows + tid * 16);
  }
  if (tid == 0) {
    if (append && ret_len < ap.retained_storage) ap.br_len[sh] = ret_len + 1;
    if (ap.window_tokens > 0 && !ap.ring_later) {
      // the ring counters belong to the sequence: the last of its heads to get here advances them
      __threadfence();
      int* seq_ticket = prm.tickets + (size_t)prm.S * prm.H + s;
      if (atomicAdd(seq_ticket, 1) == prm.H - 1) {
        *seq_ticket = 0;
        if (append) {
          if (full)
            ap.nw_pos[s] = (ring_pos + 1) % ap.window_tokens;
          else
            ap.nw_len[s] = ring_len + 1;
        }
      }
    }
  }
}

// Separate merge launch for callers whose workspace carries no tickets: one block of D threads
// per (sequence, head).
template <int D, int NQ, bool FP16>
__global__ void __launch_bounds__(D)
decode_merge_kernel(const DecodeParams prm) {
  const int sh = blockIdx.x;
  const int s = sh / prm.H, h = sh % prm.H;
  int n_total = 0;
  for (int x = 0; x < prm.n_segments; ++x) n_total += live_rows(prm.seg[x], s, h, prm.H);
  merge_records<D, NQ, FP16>(prm, sh, s, h, n_total, threadIdx.x, D);
}

}  // namespace spsattn
