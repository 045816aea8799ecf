// The launches of one decode step around the attention: the projections for a handful of rows
// (Y[r, f] = sum_k X[r, k] W[f, k], at most 16 rows, bf16, fp32 accumulation), each fused with what
// stands before and after it in the block (RMSNorm of the input; rotary embedding and the split into
// q, k, v; SwiGLU; residual add and the squares that the next RMSNorm needs), and the start of the
// step (choice of the token, counters, embedding).
//
// Bound: HBM, every weight is read once, and below that latency: a model of 12 layers and 768
// columns reads 14 MB per layer (2.2 us), so what counts is how long a launch takes to its first
// product.  Hence
//   * the launches of a step are programmatic dependents of one another: a block asks for its first
//     weights before it waits for the kernel before it;
//   * 8 features per warp, so that even 768 features occupy 96 SMs; four loader warps keep a ring of
//     shared memory full with asynchronous 16-byte copies (bulk copies of row pieces reached a sixth
//     of the bandwidth);
//   * mma.sync m16n8k16 with the rows on the M side, fragments read from shared memory with 8 bytes
//     per lane (rows are padded to 32 bytes past a multiple of 128: no bank conflicts; a lane's four
//     elements are neighbours, as the order inside the 16 columns of one product is free).
//     tcgen05 was slower here (25-45 clk to issue each product of M = 64, a commit and a read of
//     tensor memory at the end: 490 against 375 us for a token of the model above when it was tried;
//     295 now, 566 with library projections and separate kernels).
// The contraction of one output is one chain of products, sixteen columns at a time in ascending k, never split, with results
// rounded to bf16 where the separate kernels (library GEMM, model_glue.cuh, rope.cuh) round theirs and
// the norm's sums in the order of add_rmsnorm_kernel.  A step's logits were the same bits as theirs at nine
// of eleven sizes with CUDA 12.9's library; at vocabularies of 1001 and 9473, where the library takes another
// algorithm for the head, 2e-6 and 1e-4 of their norm apart.  (Rounding flips spread: with the contraction split over eight warps the logits of a 24-layer model
// moved by 3 % of their norm.)
#pragma once

#include "common.cuh"
#include "model_glue.cuh"

namespace spsattn {

enum SkinnyEpilogue { kSkinnyQkv = 0, kSkinnyResidual = 1, kSkinnySwiglu = 2, kSkinnyLogits = 3 };
// Taken up to 8 rows, of narrow steps up to 16, and where the projections of decoder_rows.cuh do not take the
// sizes (rows_faster has both sides measured); for the head.
constexpr int kSkinnyMaxRows = 16;
constexpr int kSkinnyMaxCols = 2048;   // of a normalised input: one vector of 8 per thread of add_rmsnorm_kernel
constexpr int kSkinnyMaxStages = 16;
constexpr int kSkinnyMaxWarps = 12;    // that multiply
constexpr int kSkinnyLoaders = 128;    // threads that copy
constexpr int kSkinnyMinThreads = 256; // blocks with fewer tiles still stage their input with this many

struct SkinnyParams {
  const uint16_t* w;         // [F, K]; SwiGLU: [2F, K], gate rows then up rows
  const uint16_t* x;         // row r at x + r * x_stride
  int64_t x_stride;
  int K, F, rows;            // F: outputs per row
  int warps;                 // multiplying warps per block, 8 outputs each per round
  int kc, stages;            // columns per stage of the ring
  // RMSNorm of the input rows: part i of row r (ssq[r * ssq_stride + i]) is the sum of squares of
  // its elements 8i .. 8i+7
  const uint16_t* norm_w;
  const float* ssq;
  int64_t ssq_stride;
  float eps;
  uint16_t* out;             // SwiGLU, logits: [rows, F]; residual: x in place
  float* ssq_out;            // residual: [rows, F / 8]
  const int8_t* active;      // [batch]; logits: rows with 0 are written as zeros
  // q, k, v: rows are (sequence, slot); q [rows, C], k and v [slots, batch, C]
  uint16_t *q, *k, *v;
  const float2* freqs;       // [positions, head_dim / 2] (cos, sin)
  const int64_t* pos;        // [batch]
  int slots, batch, head_dim;
  // residual behind an attention that left it to this launch: the ring counters [batch] of the layer
  // move on (all heads of that launch have read them), for sequences of `active`
  int64_t *ring_len, *ring_pos;
  int ring_tokens;
  // logits, if the next token is chosen on the device: the largest choice_key of each row, by atomic
  // maximum (the start of the step set them to 0); ids whose bit in `suppressed` is set are not chosen
  unsigned long long* best;  // [rows] or null
  const uint32_t* suppressed;
  int* status;
};

__host__ __device__ constexpr int skinny_pitch(int columns) { return (columns * 2 + 127) / 128 * 128 + 32; }
__host__ __device__ constexpr int skinny_tile_rows(int epi) { return epi == kSkinnySwiglu ? 16 : 8; }

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint2 lds8(uint32_t addr) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  return v;
}

// one arrival when every copy that this thread has asked for so far is complete
__device__ __forceinline__ void copies_arrive(uint32_t bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}

// two bf16 of a row scaled as model_glue.cuh does: round(round(x * scale) * weight)
__device__ __forceinline__ uint32_t norm_pair(uint32_t x, uint32_t w, float scale) {
  float x0, x1, w0, w1;
  unpack2<false>(x, x0, x1);
  unpack2<false>(w, w0, w1);
  unpack2<false>(pack2<false>(x0 * scale, x1 * scale), x0, x1);
  return pack2<false>(x0 * w0, x1 * w1);
}

// Greedy choice: the first maximum; a NaN counts as the maximum, as in torch.argmax.  One 64-bit key per
// logit, its order as an integer, then the complement of its index, so that the largest key is it.
// Never 0.  u: bits of the logit as fp32.
__device__ __forceinline__ unsigned long long choice_key(uint32_t u, int i, bool hidden) {
  if ((u & 0x7fffffffu) == 0) u = 0;                          // -0 equals 0
  uint32_t order = u & 0x80000000u ? ~u : u | 0x80000000u;
  if ((u & 0x7fffffffu) > 0x7f800000u) order = 0xffffffffu;   // NaN
  if (hidden) order = 0x007fffffu;                            // -inf
  return ((unsigned long long)order << 32) | (uint32_t)~(uint32_t)i;
}

// MT: tiles of 8 input rows (1 or 2)
template <int EPI, int MT>
__global__ void __launch_bounds__(32 * kSkinnyMaxWarps + kSkinnyLoaders) skinny_gemm_kernel(const SkinnyParams p) {
  constexpr bool kNorm = EPI != kSkinnyResidual;
  constexpr int R = skinny_tile_rows(EPI);         // weight rows per tile
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t s_full[kSkinnyMaxStages], s_empty[kSkinnyMaxStages];
  __shared__ int s_abort;
  __shared__ float s_scale[kSkinnyMaxRows];
  __shared__ unsigned long long s_best[kSkinnyMaxRows];    // logits
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int threads = blockDim.x, loader = tid - (threads - kSkinnyLoaders);     // below 0: not one
  const int g = lane >> 2, t = lane & 3;
  grid_launch_dependents();

  const uint32_t smem = smem_u32(smem_raw);
  const int pitch = skinny_pitch(p.kc);
  const int w_bytes = p.warps * R * pitch;
  const int stage_bytes = w_bytes + (kNorm ? 0 : p.rows * pitch);
  const uint32_t s_x = smem + p.stages * stage_bytes;      // normalised input rows
  const int x_pitch = kNorm ? skinny_pitch(p.K) : pitch;
  const uint32_t full0 = smem_u32(s_full), empty0 = smem_u32(s_empty);
  const int chunks = (p.K + p.kc - 1) / p.kc;
  const int per_round = 8 * p.warps;               // outputs of one block in one round
  const int rounds_all = (p.F + per_round - 1) / per_round;
  const int rounds = (rounds_all - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  volatile int* abort_flag = &s_abort;

  // One stage: row pieces of kc columns (of the last chunk: what is left), 16 bytes per copy, the
  // loaders' lanes along a row.  kc <= 1024: one vector of a row per loader at most.
  const int vecs_kc = p.kc / 8, row_step = kSkinnyLoaders / vecs_kc;
  const int my_row = loader / vecs_kc, my_vec = loader - my_row * vecs_kc;
  auto load_weights = [&](int st, int f0, int j) {
    const int vecs = min(p.kc, p.K - j * p.kc) / 8, have = min(per_round, p.F - f0);
    const uint32_t dst = smem + st * stage_bytes + my_vec * 16;
    const uint16_t* src = p.w + (size_t)f0 * p.K + j * p.kc + my_vec * 8;
    if (my_vec < vecs) {
      if constexpr (EPI == kSkinnySwiglu) {
        const size_t up = (size_t)p.F * p.K;
        for (int o = my_row; o < have; o += row_step) {
          const uint32_t at = dst + ((o >> 3) * 16 + (o & 7)) * pitch;
          copy16(at, src + (size_t)o * p.K);
          copy16(at + 8 * pitch, src + up + (size_t)o * p.K);
        }
      } else {
        for (int o = my_row; o < have; o += row_step) copy16(dst + o * pitch, src + (size_t)o * p.K);
      }
    }
    copies_arrive(full0 + 8 * st);
  };
  auto load_rows = [&](int st, int j) {
    const int vecs = min(p.kc, p.K - j * p.kc) / 8;
    if (my_vec < vecs)
      for (int r = my_row; r < p.rows; r += row_step)
        copy16(smem + st * stage_bytes + w_bytes + r * pitch + my_vec * 16, p.x + r * p.x_stride + j * p.kc + my_vec * 8);
    copies_arrive(full0 + 8 * st);
  };

  const int loads = rounds * chunks, first = min(loads, p.stages);
  if (EPI == kSkinnyLogits && tid < kSkinnyMaxRows) s_best[tid] = 0;
  if (loader == 0) {
    s_abort = 0;
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(full0 + 8 * i, kNorm ? kSkinnyLoaders : 2 * kSkinnyLoaders);    // weights (and input rows)
      mbar_init(empty0 + 8 * i, p.warps);
    }
    fence_barrier_init();
  }
  if (loader >= 0) {
    asm volatile("bar.sync 1, %0;" ::"n"(kSkinnyLoaders) : "memory");
    for (int n = 0, j = 0, it = 0; n < first; ++n) {
      load_weights(n, ((int)blockIdx.x + it * (int)gridDim.x) * per_round, j);
      if (++j == chunks) j = 0, ++it;
    }
  }

  // ------------------------------------------------------------------ input rows
  int64_t pos[MT] = {};                // of the lane's rows (q, k, v)
  // q, k, v: which of them output f belongs to and its pair inside a head; the remainder of the first
  // round is taken before the wait
  const int C = EPI == kSkinnyQkv ? p.F / 3 : 1;
  auto part_of = [&](int f) { return EPI == kSkinnyQkv ? (f >= C) + (f >= 2 * C) : 0; };
  auto pair_of = [&](int f) { return EPI == kSkinnyQkv ? (f - part_of(f) * C) % p.head_dim / 2 : 0; };
  const int first_pair = pair_of((int)blockIdx.x * per_round + warp * 8 + 2 * t);
  const int two = p.slots - 1;         // rows of a sequence: 1 or 2
  if constexpr (kNorm) {
    // a thread takes one vector of 8 columns (at most 256 of them) of every `at_once`-th row
    constexpr int kOwn = 4;            // rows a thread has in flight
    const int vecs = p.K / 8, at_once = threads / vecs;
    const int sub = tid / vecs, i = tid - sub * vecs;
    const bool mine = sub < at_once;
    uint4 own[kOwn], wgt = make_uint4(0, 0, 0, 0);
    if (mine) wgt = __ldg(reinterpret_cast<const uint4*>(p.norm_w + i * 8));
    grid_dependency_wait();
    // (asked for here so that the rotary factors can be asked for as soon as the products start)
    if (EPI == kSkinnyQkv && warp < p.warps) {
#pragma unroll
      for (int m = 0; m < MT; ++m) pos[m] = g + 8 * m < p.rows ? __ldcg(p.pos + ((g + 8 * m) >> two)) : 0;
    }
    const uint16_t* xp = p.x + (size_t)sub * p.x_stride + i * 8;
    const int64_t x_step = (int64_t)at_once * p.x_stride;
#pragma unroll
    for (int k = 0; k < kOwn; ++k)
      if (mine && sub + k * at_once < p.rows) own[k] = __ldcg(reinterpret_cast<const uint4*>(xp + k * x_step));
    for (int r = warp; r < p.rows; r += threads >> 5) {
      // the order of add_rmsnorm_kernel: 256 threads with one vector each, a butterfly per 32,
      // then the eight warps in turn
      float part[8], sum = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) part[w] = w * 32 + lane < vecs ? __ldcg(p.ssq + r * p.ssq_stride + w * 32 + lane) : 0.f;
      auto butterfly = [&](int from) {       // four at a time: rows of up to 1024 columns have no more
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
          for (int w = from; w < from + 4; ++w) part[w] += __shfl_xor_sync(0xffffffffu, part[w], o);
      };
      butterfly(0);
      if (vecs > 128) butterfly(4);
#pragma unroll
      for (int w = 0; w < 8; ++w) sum += part[w];
      if (lane == 0) s_scale[r] = rsqrtf(sum / (float)p.K + p.eps);
    }
    __syncthreads();
    for (int k0 = 0; k0 * at_once < p.rows; k0 += kOwn) {
#pragma unroll
      for (int k = 0; k < kOwn; ++k) {
        const int r = sub + (k0 + k) * at_once;
        if (mine && r < p.rows) {
          const uint4 v = k0 == 0 ? own[k] : __ldcg(reinterpret_cast<const uint4*>(xp + (k0 + k) * x_step));
          const float sc = s_scale[r];
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(s_x + r * x_pitch + i * 16),
                       "r"(norm_pair(v.x, wgt.x, sc)), "r"(norm_pair(v.y, wgt.y, sc)), "r"(norm_pair(v.z, wgt.z, sc)),
                       "r"(norm_pair(v.w, wgt.w, sc))
                       : "memory");
        }
      }
    }
  } else {
    grid_dependency_wait();
    if (p.ring_len != nullptr && blockIdx.x == gridDim.x - 1 && tid < p.batch && p.active[tid] != 0) {
      const int64_t len = p.ring_len[tid], at = p.ring_pos[tid];
      if (len >= p.ring_tokens)
        p.ring_pos[tid] = (at + 1) % p.ring_tokens;
      else
        p.ring_len[tid] = len + 1;
    }
    if (loader >= 0)
      for (int n = 0, j = 0; n < first; ++n) {
        load_rows(n, j);
        if (++j == chunks) j = 0;
      }
  }
  __syncthreads();

  if (loader >= 0) {
    // ------------------------------------------------------------------ the rest of the weights
    int st = first == p.stages ? 0 : first, phase = 0, j = first % chunks, it = first / chunks;
    for (int n = first; n < loads; ++n) {
      if (!warp_wait(empty0 + 8 * st, phase, abort_flag, p.status)) break;
      load_weights(st, ((int)blockIdx.x + it * (int)gridDim.x) * per_round, j);
      if constexpr (!kNorm) load_rows(st, j);
      if (++st == p.stages) st = 0, phase ^= 1;
      if (++j == chunks) j = 0, ++it;
    }
  } else if (warp < p.warps) {
    // ------------------------------------------------------------------ products
    int st = 0, phase = 0;
    unsigned long long best[MT] = {};
    for (int it = 0; it < rounds; ++it) {
      // lane (g, t): rows g and g + 8, outputs f and f + 1
      const int f = ((int)blockIdx.x + it * (int)gridDim.x) * per_round + warp * 8 + 2 * t;
      // what the epilogue needs besides the sums is asked for here
      uint32_t old[MT], hide = 0;
      float2 cs[MT];
      if (EPI == kSkinnyLogits && p.suppressed != nullptr && f < p.F) hide = __ldg(p.suppressed + (f >> 5)) >> (f & 31);
      const int which = part_of(f), fi = f - which * C;
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const int r = g + 8 * m;
        old[m] = 0;
        cs[m] = make_float2(1.f, 0.f);
        if (r < p.rows && f < p.F) {
          if constexpr (EPI == kSkinnyResidual) old[m] = __ldcg(reinterpret_cast<const uint32_t*>(p.out + (size_t)r * p.F + f));
          if constexpr (EPI == kSkinnyQkv) {
            if (which < 2) cs[m] = __ldg(p.freqs + pos[m] * (p.head_dim / 2) + (it == 0 ? first_pair : pair_of(f)));
          }
        }
      }
      float c[R / 8][4];
#pragma unroll
      for (int x = 0; x < R / 8; ++x)
#pragma unroll
        for (int e = 0; e < 4; ++e) c[x][e] = 0.f;
      for (int j = 0; j < chunks; ++j) {
        // (a wait that gives up does not leave the loop: the waits after it return at once, and the warp
        // stays whole without a vote per stage; what is stored then is wrong, and the status word says so)
        mbar_wait(full0 + 8 * st, phase, abort_flag, p.status);
        __syncwarp();
        const uint32_t wb = smem + st * stage_bytes + (warp * R + g) * pitch + t * 8;
        const uint32_t xb = (kNorm ? s_x + j * p.kc * 2 : smem + st * stage_bytes + w_bytes) + t * 8;
        const uint32_t xa[2] = {xb + min(g, p.rows - 1) * x_pitch, xb + min(g + 8, p.rows - 1) * x_pitch};
        const int steps = min(p.kc, p.K - j * p.kc) / 16;
        // fragments of eight steps are read while the eight before them multiply (four: 6 % slower);
        // the reads carry no condition (rows past the last repeat it and reach no output)
        constexpr int U = 8;
        struct Fragments {
          uint2 a[U][MT], b[U][R / 8];
        };
        auto read = [&](Fragments& fr, int k0) {
#pragma unroll
          for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int m = 0; m < MT; ++m) fr.a[u][m] = lds8(xa[m] + (k0 + u) * 32);
#pragma unroll
            for (int x = 0; x < R / 8; ++x) fr.b[u][x] = lds8(wb + x * 8 * pitch + (k0 + u) * 32);
          }
        };
        auto multiply = [&](const Fragments& fr) {
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int x = 0; x < R / 8; ++x)
              mma_bf16_16816(c[x], fr.a[u][0].x, MT == 2 ? fr.a[u][MT - 1].x : 0u, fr.a[u][0].y,
                             MT == 2 ? fr.a[u][MT - 1].y : 0u, fr.b[u][x].x, fr.b[u][x].y);
        };
        const int whole = steps / (2 * U) * (2 * U);
        Fragments f0, f1;
        if (whole > 0) read(f0, 0);
        for (int k0 = 0; k0 < whole; k0 += 2 * U) {
          read(f1, k0 + U);
          multiply(f0);
          if (k0 + 2 * U < whole) read(f0, k0 + 2 * U);
          multiply(f1);
        }
        for (int k = whole; k < steps; ++k) {
          uint2 a[MT];
#pragma unroll
          for (int m = 0; m < MT; ++m) a[m] = lds8(xa[m] + k * 32);
#pragma unroll
          for (int x = 0; x < R / 8; ++x) {
            const uint2 b = lds8(wb + x * 8 * pitch + k * 32);
            mma_bf16_16816(c[x], a[0].x, MT == 2 ? a[MT - 1].x : 0u, a[0].y, MT == 2 ? a[MT - 1].y : 0u, b.x, b.y);
          }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(empty0 + 8 * st);
        if (++st == p.stages) st = 0, phase ^= 1;
      }

#pragma unroll
      for (int m = 0; m < MT; ++m) {
        const int r = g + 8 * m;
        const bool live = r < p.rows && f < p.F;
        float v0 = round_bf16(c[0][2 * m]), v1 = round_bf16(c[0][2 * m + 1]);
        if constexpr (EPI == kSkinnyQkv) {
          if (live) {
            if (which < 2) {
              const float a = v0, b = v1;
              v0 = __fsub_rn(__fmul_rn(a, cs[m].x), __fmul_rn(b, cs[m].y));
              v1 = __fadd_rn(__fmul_rn(a, cs[m].y), __fmul_rn(b, cs[m].x));
            }
            const int bi = r >> two, slot = r & two;
            uint16_t* dst = which == 0 ? p.q + (size_t)r * C
                                       : (which == 1 ? p.k : p.v) + ((size_t)slot * p.batch + bi) * C;
            *reinterpret_cast<uint32_t*>(dst + fi) = pack2<false>(v0, v1);
          }
        } else if constexpr (EPI == kSkinnySwiglu) {
          const float u0 = round_bf16(c[R / 8 - 1][2 * m]), u1 = round_bf16(c[R / 8 - 1][2 * m + 1]);
          if (live)
            *reinterpret_cast<uint32_t*>(p.out + (size_t)r * p.F + f) =
                pack2<false>(round_bf16(silu_f(v0)) * u0, round_bf16(silu_f(v1)) * u1);
        } else if constexpr (EPI == kSkinnyResidual) {
          float o0, o1;
          unpack2<false>(old[m], o0, o1);
          v0 = round_bf16(o0 + v0);
          v1 = round_bf16(o1 + v1);
          if (live) *reinterpret_cast<uint32_t*>(p.out + (size_t)r * p.F + f) = pack2<false>(v0, v1);
          // squares of the tile's eight elements, one after the other
          float sq = 0.f;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float e0 = __shfl_sync(0xffffffffu, v0, (lane & ~3) + q), e1 = __shfl_sync(0xffffffffu, v1, (lane & ~3) + q);
            sq = fmaf(e0, e0, sq);
            sq = fmaf(e1, e1, sq);
          }
          if (live && t == 0) p.ssq_out[(size_t)r * (p.F / 8) + f / 8] = sq;
        } else if (live) {
          const bool on = p.active == nullptr || p.active[r] != 0;
          uint16_t* dst = p.out + (size_t)r * p.F + f;
          const uint32_t both = on ? pack2<false>(v0, v1) : 0u;
          if (p.best != nullptr && on) {
            const unsigned long long k0 = choice_key(__float_as_uint(v0), f, hide & 1u);
            const unsigned long long k1 = f + 1 < p.F ? choice_key(__float_as_uint(v1), f + 1, hide & 2u) : 0;
            best[m] = max(best[m], max(k0, k1));
          }
          if (p.F % 2 == 0) {
            *reinterpret_cast<uint32_t*>(dst) = both;
          } else {
            dst[0] = (uint16_t)both;
            if (f + 1 < p.F) dst[1] = (uint16_t)(both >> 16);
          }
        }
      }
    }
    if (EPI == kSkinnyLogits && p.best != nullptr) {
      // one atomic per block and row: 1776 warps on one address would queue for longer than they multiply
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        best[m] = max(best[m], __shfl_xor_sync(0xffffffffu, best[m], 1));
        best[m] = max(best[m], __shfl_xor_sync(0xffffffffu, best[m], 2));
        if (t == 0 && g + 8 * m < p.rows) atomicMax(&s_best[g + 8 * m], best[m]);
      }
      asm volatile("bar.sync 2, %0;" ::"r"(32 * p.warps) : "memory");
      if (tid < p.rows && s_best[tid] != 0) atomicMax(p.best + tid, s_best[tid]);
    }
  }
  // a step that was given up may leave copies in flight
  if (loader >= 0) asm volatile("cp.async.wait_all;" ::: "memory");
}

// ---------------------------------------------------------------------------------------------
// Start of a decode step, one block per sequence: choose the token (greedy over the logits of the
// step before, or the caller's), book-keeping of the sequence's counters, embedding of its rows.
// Stands in for two dozen small launches of the same steps in tensor operations, which cost more
// than the projections of a small model.  Bound: latency, a chain of dependent reads.  The choice is
// left by the head of the step before (SkinnyParams::best): reading 50304 logits again took the block
// 11 of its 14 us.  They are read here only behind the prefill and behind library projections.
struct TokenStartParams {
  // greedy choice (logits null: tokens and activity come from token_in / active_in)
  const void* logits;            // [batch, vocab] bf16 or fp32
  const uint32_t* suppressed;    // bit per token id, or null
  int64_t* generated;            // [batch, max_new], written at *step
  int64_t* step;                 // [batch] tokens chosen so far (advanced here)
  uint8_t* finished;             // [batch]
  unsigned long long* best;      // [batch] largest choice_key of the row, 0: not known; or null
  int max_new, stop_on_eos;
  int choose_only;               // the last token: nothing is embedded or advanced
  const int64_t* token_in;       // [batch]
  const uint8_t* active_in;      // [batch]
  // sequence state
  int64_t* processed;            // [batch]
  uint8_t* next_doc_start;       // [batch]
  int64_t *nw_len, *nw_pos;      // [layers, batch]
  int64_t* br_len;               // [layers, batch, heads]
  int layers, batch, heads, vocab;
  int64_t eos, pad, predict;
  // outputs of the step's first launches
  int8_t* active;                // [batch]
  int64_t* pos;                  // [batch]
  const float2* freqs;           // [positions, half_dim] (cos, sin)
  float2* freqs_out;             // [batch, half_dim]: the sequence's row, or null
  int half_dim;
  const void* wte;               // [vocab, C] bf16 or fp32
  int wte_wide;                  // 16-byte aligned
  void* x;                       // [batch * slots, C]
  float* ssq;                    // [batch * slots, C / 8] sums of squares of 8 elements each, or null (bf16 only)
  int slots, C;
  int* status;
};

constexpr int kStartThreads = 1024;

template <bool F32>
__global__ void __launch_bounds__(kStartThreads) token_start_kernel(const TokenStartParams p) {
  __shared__ unsigned long long s_best[kStartThreads / 32];
  const int b = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // Dependents are let go only after the wait: what they touch before their own wait (weights) is
  // then no longer being written by anything before this step.
  grid_dependency_wait();
  grid_launch_dependents();

  // All threads read the sequence's state and come to the same choice; thread 0 writes it back at the end.
  const int64_t n = p.choose_only ? 0 : p.processed[b];
  const bool starts_doc = !p.choose_only && p.next_doc_start[b] != 0;
  bool live, newly = false;
  int64_t chosen, at = 0;
  if (p.logits != nullptr) {
    live = p.finished[b] == 0;
    at = p.step[b];
    unsigned long long best = p.best == nullptr ? 0 : __ldcg(p.best + b);
    if (live && best == 0) {
      auto take = [&](uint32_t u, int i, uint32_t hidden) { best = max(best, choice_key(u, i, hidden != 0)); };
      constexpr int V = F32 ? 4 : 8, U = 4;    // logits per 16-byte load, loads in flight
      const uint8_t* row = reinterpret_cast<const uint8_t*>(p.logits) + (size_t)b * p.vocab * (F32 ? 4 : 2);
      if (p.vocab % V == 0) {
        for (int i0 = tid; i0 < p.vocab / V; i0 += U * kStartThreads) {
          uint4 u[U];
          uint32_t hide[U];
#pragma unroll
          for (int x = 0; x < U; ++x) {
            const int i = i0 + x * kStartThreads;
            if (i < p.vocab / V) {
              u[x] = __ldcg(reinterpret_cast<const uint4*>(row) + i);
              hide[x] = p.suppressed == nullptr ? 0u : p.suppressed[i * V >> 5] >> (i * V & 31);
            }
          }
#pragma unroll
          for (int x = 0; x < U; ++x) {
            const int i = i0 + x * kStartThreads;
            if (i < p.vocab / V) {
              const uint32_t w[4] = {u[x].x, u[x].y, u[x].z, u[x].w};
#pragma unroll
              for (int e = 0; e < V; ++e)
                take(F32 ? w[e * 4 / V] : e & 1 ? w[e * 4 / V] & 0xffff0000u : w[e * 4 / V] << 16, i * V + e, (hide[x] >> e) & 1u);
            }
          }
        }
      } else {
        for (int i = tid; i < p.vocab; i += kStartThreads)
          take(F32 ? reinterpret_cast<const uint32_t*>(row)[i] : (uint32_t)reinterpret_cast<const uint16_t*>(row)[i] << 16, i,
               p.suppressed == nullptr ? 0u : (p.suppressed[i >> 5] >> (i & 31)) & 1u);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
      if (lane == 0) s_best[warp] = best;
      __syncthreads();
      best = s_best[lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
    }
    chosen = live ? (int64_t)(uint32_t)~(uint32_t)best : p.pad;
    newly = live && p.stop_on_eos && chosen == p.eos;
    if (p.choose_only) {
      if (tid == 0 && at < p.max_new) p.generated[(size_t)b * p.max_new + at] = chosen;
      return;
    }
  } else {
    chosen = p.token_in[b];
    live = p.active_in[b] != 0;
  }
  // A caller's id outside the vocabulary is reported, and its sequence sits the step out.
  const bool wanted = live && !newly;
  const bool known = chosen >= 0 && chosen < p.vocab && (p.slots == 1 || (p.predict >= 0 && p.predict < p.vocab));
  const bool active = wanted && known;
  const int64_t token = active ? chosen : 0;
  if (wanted && !known && tid == 0 && p.status != nullptr) atomicOr(p.status, SPSATTN_STATUS_BAD_TOKEN);

  // a row that starts a document forgets its caches, in every layer
  if (active && starts_doc) {
    for (int i = tid; i < p.layers * p.heads; i += kStartThreads)
      p.br_len[((size_t)(i / p.heads) * p.batch + b) * p.heads + i % p.heads] = 0;
    for (int i = tid; i < p.layers; i += kStartThreads) {
      p.nw_len[(size_t)i * p.batch + b] = 0;
      p.nw_pos[(size_t)i * p.batch + b] = 0;
    }
  }
  constexpr int V = F32 ? 4 : 8;
  for (int idx = tid; idx < p.slots * (p.C / V); idx += kStartThreads) {
    const int slot = idx / (p.C / V), i = idx - slot * (p.C / V);
    const int64_t id = slot == 0 ? token : p.predict;
    uint4 u = make_uint4(0, 0, 0, 0);
    if (id >= 0 && id < p.vocab) {
      const size_t at = (size_t)id * (p.C / V) + i;
      if (p.wte_wide) {
        u = reinterpret_cast<const uint4*>(p.wte)[at];
      } else if constexpr (F32) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(p.wte) + at * V;
        u = make_uint4(w[0], w[1], w[2], w[3]);
      } else {
        const uint16_t* w = reinterpret_cast<const uint16_t*>(p.wte) + at * V;
        u = make_uint4(w[0] | (uint32_t)w[1] << 16, w[2] | (uint32_t)w[3] << 16, w[4] | (uint32_t)w[5] << 16,
                       w[6] | (uint32_t)w[7] << 16);
      }
    }
    reinterpret_cast<uint4*>(p.x)[((size_t)b * p.slots + slot) * (p.C / V) + i] = u;
    if (!F32 && p.ssq != nullptr) {
      float f[8], sq = 0.f;
      unpack2<false>(u.x, f[0], f[1]);
      unpack2<false>(u.y, f[2], f[3]);
      unpack2<false>(u.z, f[4], f[5]);
      unpack2<false>(u.w, f[6], f[7]);
#pragma unroll
      for (int e = 0; e < 8; ++e) sq = fmaf(f[e], f[e], sq);
      p.ssq[((size_t)b * p.slots + slot) * (p.C / 8) + i] = sq;
    }
  }
  if (p.freqs_out != nullptr)
    for (int i = tid; i < p.half_dim; i += kStartThreads)
      p.freqs_out[(size_t)b * p.half_dim + i] = p.freqs[(active ? n : 0) * p.half_dim + i];
  __syncthreads();               // everybody has read the state
  if (tid == 0) {
    if (p.logits != nullptr) {
      if (at < p.max_new) p.generated[(size_t)b * p.max_new + at] = chosen;
      p.step[b] = at + 1;
      if (newly) p.finished[b] = 1;
      if (p.best != nullptr) p.best[b] = 0;
    }
    p.active[b] = active ? 1 : 0;
    p.pos[b] = active ? n : 0;
    if (active) {
      p.processed[b] = n + 1;
      p.next_doc_start[b] = chosen == p.eos ? 1 : 0;
    }
  }
}

}  // namespace spsattn
