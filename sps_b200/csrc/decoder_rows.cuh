// The projections of a decode step of 9 to 64 rows (wide models: of 1 to 64): Y[r, f] = sum_k X[r, k] W[f, k], bf16, fp32
// accumulation, each with what stands behind it in the block (rotary embedding and the split into
// q, k, v; residual add; SwiGLU).
//
// Bound: HBM (every weight is read once), and at small widths the latency of the launches.  Library
// products of 64 rows reached half of the copy bandwidth (gate/up of 2048 -> 2 x 8192: 13.0 us, 10.3 at the
// copy bandwidth; q/k/v 7.2, 3.9), and the element-wise kernels behind them cost 2.7 us each.  Hence
//   * one block per `bn` weight rows and `bm` input rows, sized so that a projection is one wave: the
//     weights are the N side of tcgen05.mma (any multiple of 8), the rows its M = 64;
//   * TMA brings both operands, up to 512 columns a stage (one copy each), through a ring as deep as shared
//     memory allows: with 64 columns a stage the waits and issues around a stage took 430 clk, its products 124
//     (2048 x 8192: 34 us);
//   * the launches of a step are programmatic dependents of one another: a block asks for its whole ring
//     of weights before it waits for the kernel before it, the input rows follow after the wait;
//   * tensor memory is allocated after that wait: a block that held some while the attention before it
//     still had blocks without theirs would wait for them, and they for it.
// us per token, captured, two rows per sequence, library projections with single kernels / now: 12 layers of 768 columns
// 18 rows 449 / 320, 32 rows 463 / 322; 12 x 1024, 32 rows 505 / 357; 6 x 2048, 24 rows 385 / 322, 64 rows 469 / 422.
// What is left at 2048 columns: 31 clk per 16 columns of a chain (2048 x 8192: 512 of them, 8 us), 300 clk per stage.
// The contraction of one output is one chain of products in ascending k, never split, rounded to bf16 where
// the separate kernels (library product, model_glue.cuh, rope.cuh) round theirs: the same bits as theirs at every
// size compared (up to 24 layers of 2048 columns, 9 to 64 rows).
#pragma once

#include "common.cuh"
#include "decoder_rows_ring.h"
#include "model_glue.cuh"

namespace spsattn {

enum RowsEpilogue { kRowsQkv = 0, kRowsResidual = 1, kRowsSwiglu = 2 };
constexpr int kRowsMaxRows = 64;
constexpr int kRowsThreads = 192;      // four warps of the epilogue, loads, products
constexpr int kRowsMaxStages = 24;
constexpr int kRowsMaxN = 128;         // weight rows per block
constexpr int kRowsHeldN = 64;         // the same where the epilogue holds operands of its own in registers

struct RowsGemmParams {
  int K, F, rows;            // F: outputs per row
  int bn, bm;                // weight rows (SwiGLU: half gate, half up) and input rows per block
  int stages, groups;        // of the ring; groups of 64 columns per stage
  uint16_t* out;             // SwiGLU: [rows, F]; residual: [rows, F], x in place
  // q, k, v: rows are (sequence, slot); q [rows, C], k and v [slots, batch, C]
  uint16_t *q, *k, *v;
  const float2* freqs;       // [batch, head_dim / 2] (cos, sin) of the sequences' positions
  int slots, batch, head_dim;
  float* ssq_out;            // residual: [rows, F / 8] sums of squares of 8 elements of the new row, or null
  // residual behind an attention that left it to this launch: the ring counters [batch] of the layer
  // move on (all heads of that launch have read them), for sequences of `active`
  int64_t *ring_len, *ring_pos;
  const int8_t* active;
  int ring_tokens;
  int* status;
};

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

// umma_ss that starts the sums or goes on with them
__device__ __forceinline__ void umma_ss_if(uint32_t d_tmem, uint32_t a_lo, uint32_t a_hi, uint32_t b_lo, uint32_t b_hi,
                                           uint32_t idesc, bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.u32 p, %6, 0;\n\t"
      "mov.b64 da, {%1, %2};\n\t"
      "mov.b64 db, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}"
      ::"r"(d_tmem), "r"(a_lo), "r"(a_hi), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}

// A wait expired, of whichever warp of the block: no copy and no product stays in flight when its memory is given
// up.  (A function of its own, and the loops over groups are not unrolled: the instructions of a launch come from
// caches that do not have them yet.  12 layers of 768 columns, 16 rows, us per token: without this 328, with it on
// every launch's way 342, so 338, with those loops short as well 314.)
__device__ __noinline__ void rows_give_up(uint32_t full0, int asked, int stages, uint32_t products) {
  int unused = 0;
  rows_landed(asked, stages, [&](int st, int phase) { mbar_wait(full0 + 8 * st, phase, &unused, nullptr); });
  mbar_wait(products, 0, &unused, nullptr);
}

template <int EPI>
__global__ void __launch_bounds__(kRowsThreads, 1)
rows_gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_x,
                 const __grid_constant__ RowsGemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t s_full[kRowsMaxStages], s_empty[kRowsMaxStages], s_done, s_quit;
  __shared__ uint32_t s_tmem;
  __shared__ int s_abort, s_asked, s_stopped;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  grid_launch_dependents();
  const uint32_t smem = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t full0 = smem_u32(s_full), empty0 = smem_u32(s_empty), done = smem_u32(&s_done), quit = smem_u32(&s_quit);
  const int x_sub = p.bm * 128, x_bytes = p.groups * x_sub;       // 64 columns of the input rows; a stage of them
  const int w_sub = p.bn * 128;
  const int stage_bytes = x_bytes + p.groups * w_sub;
  const int all_groups = p.K / 64, chunks = (all_groups + p.groups - 1) / p.groups, first = min(chunks, p.stages);
  const int bf = EPI == kRowsSwiglu ? p.bn / 2 : p.bn;            // outputs of a row per block
  const int f0 = blockIdx.x * bf, r0 = blockIdx.y * p.bm;
  volatile int* abort_flag = &s_abort;

  auto load_w = [&](int st, int j) {                               // one elected lane
    const uint32_t dst = smem + st * stage_bytes + x_bytes;
    mbar_arrive_expect_tx(full0 + 8 * st, (uint32_t)stage_bytes);
    if constexpr (EPI == kRowsSwiglu) {
      // gate rows and up rows of 64 columns lie under one another
#pragma unroll 1
      for (int g = 0; g < p.groups; ++g) {
        tma_load_3d(dst + g * w_sub, &tm_w, full0 + 8 * st, 0, f0, j * p.groups + g);
        tma_load_3d(dst + g * w_sub + bf * 128, &tm_w, full0 + 8 * st, 0, p.F + f0, j * p.groups + g);
      }
    } else {
      tma_load_3d(dst, &tm_w, full0 + 8 * st, 0, f0, j * p.groups);
    }
  };
  auto load_x = [&](int st, int j) { tma_load_3d(smem + st * stage_bytes, &tm_x, full0 + 8 * st, 0, r0, j * p.groups); };

  if (warp == 4) {
    if (lane == 0) {
      s_abort = s_stopped = 0;
      s_asked = chunks;
      for (int i = 0; i < p.stages; ++i) {
        mbar_init(full0 + 8 * i, 1);
        mbar_init(empty0 + 8 * i, 1);
      }
      mbar_init(done, 1);
      mbar_init(quit, 1);
      fence_barrier_init();
      tma_prefetch_desc(&tm_w);
      tma_prefetch_desc(&tm_x);
    }
    __syncwarp();
    if (elect_one())
      for (int j = 0; j < first; ++j) load_w(j, j);
    __syncwarp();
  }
  grid_dependency_wait();
  if (EPI == kRowsResidual && p.ring_len != nullptr && blockIdx.x == 0 && blockIdx.y == 0 && tid < p.batch && p.active[tid] != 0) {
    const int64_t len = p.ring_len[tid], at = p.ring_pos[tid];
    if (len >= p.ring_tokens)
      p.ring_pos[tid] = (at + 1) % p.ring_tokens;
    else
      p.ring_len[tid] = len + 1;
  }
  if (warp == 4) {
    if (elect_one())
      for (int j = 0; j < first; ++j) load_x(j, j);
    __syncwarp();
  } else if (warp == 5) {
    tmem_alloc<128>(smem_u32(&s_tmem));
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s_tmem;

  if (warp == 4) {
    // ------------------------------------------------------------------ loads
    if (elect_one()) {
      const int asked = rows_feed(
          first, chunks, p.stages, [&](int st, int phase) { return mbar_wait(empty0 + 8 * st, phase, abort_flag, p.status); },
          [&](int st, int j) {
            load_w(st, j);
            load_x(st, j);
          });
      if (asked < chunks) s_asked = asked;
    }
    __syncwarp();
  } else if (warp == 5) {
    // ------------------------------------------------------------------ products
    // rows past bm of the M side are whatever follows in shared memory: an MMA row mixes with no other
    const uint32_t idesc = make_idesc_f16(false, 64, 0, false, false) | ((uint32_t)(p.bn >> 3) << 17);
    const uint64_t dx = make_smem_desc_sw128(smem, 16, 1024), dw = make_smem_desc_sw128(smem + x_bytes, 16, 1024);
    const uint32_t x_lo = (uint32_t)dx, x_hi = (uint32_t)(dx >> 32), w_lo = (uint32_t)dw, w_hi = (uint32_t)(dw >> 32);
    // One elected lane from here to the end: a step of 16 columns takes 31 clk (M = 64, up to 32 weight rows),
    // and with the whole warp around every stage (a vote, an election and a reconvergence each) a stage took
    // 300 clk more.
    if (elect_one()) {
      int st = 0, phase = 0, j = 0;
      for (; j < chunks; ++j) {
        if (!mbar_wait(full0 + 8 * st, phase, abort_flag, p.status)) break;
        tc_fence_after();
        const uint32_t xa = x_lo + ((uint32_t)(st * stage_bytes) >> 4), wa = w_lo + ((uint32_t)(st * stage_bytes) >> 4);
        const int groups = min(p.groups, all_groups - j * p.groups);
#pragma unroll 1
        for (int g = 0; g < groups; ++g) {
          const uint32_t x = xa + ((uint32_t)(g * x_sub) >> 4), w = wa + ((uint32_t)(g * w_sub) >> 4);
#pragma unroll
          for (int kk = 0; kk < 4; ++kk) umma_ss_if(tmem, x + 2 * kk, x_hi, w + 2 * kk, w_hi, idesc, j + g + kk > 0);
        }
        umma_commit(empty0 + 8 * st);
        if (j == chunks - 1) umma_commit(done);
        if (++st == p.stages) st = 0, phase ^= 1;
      }
      if (j < chunks) {
        umma_commit(quit);
        s_stopped = 1;
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ results
    // The sums go through shared memory (the ring, whose copies and products are over by then), so that all
    // threads work, each on vectors of 8 outputs of a row, and rows are written in one piece: with a row per
    // lane (16 of 32 lanes have one) and everything unrolled the results took 2000 clk, most of them for
    // instructions that no cache had yet.
    const int vecs = bf / 8, rows_here = min(p.bm, p.rows - r0), items = rows_here * vecs;
    const int two = p.slots - 1, C = EPI == kRowsQkv ? p.F / 3 : 1;
    constexpr int kHeld = EPI == kRowsSwiglu ? 1 : kRowsMaxRows * kRowsHeldN / 8 / 128;
    // what stands beside the sums is asked for while they are made: the old row, or the rotary factors
    uint4 old[EPI == kRowsResidual ? kHeld : 1];
    float4 cs[EPI == kRowsQkv ? kHeld : 1][2];
    if constexpr (EPI != kRowsSwiglu) {
#pragma unroll
      for (int k = 0; k < kHeld; ++k) {
        const int i = tid + 128 * k, rl = i / vecs, f = f0 + (i - rl * vecs) * 8, r = r0 + rl;
        if (i < items && f < p.F) {
          if constexpr (EPI == kRowsResidual) old[k] = __ldcg(reinterpret_cast<const uint4*>(p.out + (size_t)r * p.F + f));
          if constexpr (EPI == kRowsQkv) {
            if (f < 2 * C) {
              const float4* fr = reinterpret_cast<const float4*>(p.freqs + (size_t)(r >> two) * (p.head_dim / 2) + (f >= C ? f - C : f) % p.head_dim / 2);
              cs[k][0] = __ldcg(fr);
              cs[k][1] = __ldcg(fr + 1);
            }
          }
        }
      }
    }
    const bool ok = __all_sync(0xffffffffu, mbar_wait(done, 0, abort_flag, p.status));
    const int pitch = p.bn * 4 + 16;                 // bytes of a row of sums
    if (ok) {
      tc_fence_after();
      // M = 64: row r of the accumulator lies in lane 32 * (r / 16) + r % 16
      const uint32_t at = tmem + ((uint32_t)(warp * 32) << 16), to = smem + (warp * 16 + lane) * pitch;
#pragma unroll 1
      for (int c = 0; c < p.bn; c += 8) {
        uint32_t a[8];
        tmem_ld8(at + c, a);
        tmem_wait_ld();
        if (lane < 16) {
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to + c * 4), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]) : "memory");
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(to + c * 4 + 16), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(a[7]) : "memory");
        }
      }
      tc_fence_before();
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    auto sums = [&](uint32_t from, float (&v)[8]) {
      const uint4 lo = lds16(from), hi = lds16(from + 16);
      const uint32_t w[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = round_bf16(__uint_as_float(w[e]));
    };
    auto result = [&](int k) {
      const int i = tid + 128 * k, rl = i / vecs, c = (i - rl * vecs) * 8, f = f0 + c, r = r0 + rl;
      if (!ok || i >= items || f >= p.F) return;
      float v[8];
      sums(smem + rl * pitch + c * 4, v);
      uint16_t* dst;
      if constexpr (EPI == kRowsSwiglu) {
        float u[8];
        sums(smem + rl * pitch + (bf + c) * 4, u);
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = round_bf16(silu_f(v[e])) * u[e];
        dst = p.out + (size_t)r * p.F + f;
      } else if constexpr (EPI == kRowsResidual) {
        const uint32_t w[4] = {old[k].x, old[k].y, old[k].z, old[k].w};
        float sq = 0.f;
#pragma unroll
        for (int e = 0; e < 8; e += 2) {
          float o0, o1;
          unpack2<false>(w[e / 2], o0, o1);
          v[e] = round_bf16(o0 + v[e]);
          v[e + 1] = round_bf16(o1 + v[e + 1]);
          sq = fmaf(v[e], v[e], sq);
          sq = fmaf(v[e + 1], v[e + 1], sq);
        }
        if (p.ssq_out != nullptr) p.ssq_out[(size_t)r * (p.F / 8) + f / 8] = sq;
        dst = p.out + (size_t)r * p.F + f;
      } else {
        const int which = (f >= C) + (f >= 2 * C), fi = f - which * C;
        if (which < 2) {
          const float q[8] = {cs[k][0].x, cs[k][0].y, cs[k][0].z, cs[k][0].w, cs[k][1].x, cs[k][1].y, cs[k][1].z, cs[k][1].w};
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            const float x0 = v[e], x1 = v[e + 1];
            v[e] = __fsub_rn(__fmul_rn(x0, q[e]), __fmul_rn(x1, q[e + 1]));
            v[e + 1] = __fadd_rn(__fmul_rn(x0, q[e + 1]), __fmul_rn(x1, q[e]));
          }
        }
        dst = which == 0 ? p.q + (size_t)r * C + fi
                         : (which == 1 ? p.k : p.v) + ((size_t)(r & two) * p.batch + (r >> two)) * C + fi;
      }
      *reinterpret_cast<uint4*>(dst) = make_uint4(pack2<false>(v[0], v[1]), pack2<false>(v[2], v[3]), pack2<false>(v[4], v[5]),
                                                  pack2<false>(v[6], v[7]));
    };
    if constexpr (EPI == kRowsSwiglu) {
#pragma unroll 1
      for (int k = 0; 128 * k < items; ++k) result(k);
    } else {
#pragma unroll
      for (int k = 0; k < kHeld; ++k)
        if (128 * k < items) result(k);
    }
  }
  __syncthreads();
  if (*abort_flag != 0) {
    if (tid == 128) rows_give_up(full0, s_asked, p.stages, s_stopped ? quit : done);
    __syncthreads();
  }
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc<128>(tmem);
  }
}

}  // namespace spsattn
