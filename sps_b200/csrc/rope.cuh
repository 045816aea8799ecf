// Rotary embedding + cast, the producer side of the attention operands: reads q or k as the
// projection left them ([B, N, H, D] view, bf16 / fp16 / fp32, any row strides), rotates adjacent
// element pairs by the position's complex frequency in fp32 and writes 16-bit rows in the layout
// the attention kernel reads in place.  With rotate = 0 it is a plain cast (for v).
// The H heads of the view may be split into up to six consecutive groups (the q, k and v thirds
// of a fused projection; for a decode step, those of both slots of a token pair), each with its
// own destination, strides and rotate flag, so that one launch produces all operands.
// Reference computation: src/modeling/models/model.py:201-230 (apply_rotary_emb: view pairs as
// complex, multiply by freqs_cis, back to real, cast) followed by the bf16 cast of
// src/modeling/models/sps/core.py:53-55.
#pragma once

#include "common.cuh"

namespace spsattn {

constexpr int kMaxRopeGroups = 6;

struct RopeGroup {
  uint16_t* out;
  int64_t os_b, os_n, os_h;    // elements
  int rotate;
};

struct RopeParams {
  const void* x;
  int64_t xs_b, xs_n, xs_h;    // elements
  const float2* freqs;         // [N, D/2] or [B, N, D/2] (cos, sin)
  int64_t fs_b;                // elements of float2 per batch row, 0 when shared
  RopeGroup group[kMaxRopeGroups];
  int heads_per_group;         // H = n_groups * heads_per_group
  int out_fp16;
  int B, N, H, D;
  // launch: rows that a thread walks down; rows side by side in a block, and their number as batches and rows
  int walk, side, step_b, step_n;
};

// Bound: HBM.  A thread keeps its place in the row (head, group, eight elements) and walks down `walk`
// rows, two loads in flight, so that nothing is divided per element: one flat index per vector
// reached half of the bandwidth (65536 rows of 6144: 440 -> 283 us, 5.7 TB/s).
// X_DTYPE: 0 bf16, 1 fp16, 2 fp32.  kSide: many narrow rows, `side` of them next to one another in a block;
// with a row per block, 65536 rows of one head of 16 took 30 us, now 2.9 (a kernel of its own: the general
// step from row to row alone cost wide fp32 rows 20 %, 72 -> 86 us for 32768 rows of 2304).
template <int X_DTYPE, bool kSide>
__global__ void __launch_bounds__(256, 4) rope_cast_kernel(const RopeParams p) {
  grid_dependency_wait();
  const int vec_per_head = p.D / 8, vecs = p.H * vec_per_head;
  const int side = kSide ? p.side : 1, mine = kSide ? (int)threadIdx.x / vecs : 0;
  if (mine >= side) return;
  const long long row0 = (long long)blockIdx.x * p.walk * side + mine;
  const int count = (int)min((long long)p.walk, ((long long)p.B * p.N - row0 + side - 1) / side);
  const int b0 = (int)(row0 / p.N), n0 = (int)(row0 - (long long)b0 * p.N);
  constexpr int kBytes = X_DTYPE == 2 ? 4 : 2, kLoads = kBytes / 2;      // 16-byte loads per vector
  for (int v = kSide ? threadIdx.x - mine * vecs : blockIdx.y * 256 + threadIdx.x; v < vecs; v += kSide ? vecs : gridDim.y * 256) {
    const int h = v / vec_per_head, x8 = v - h * vec_per_head;
    const int gi = h / p.heads_per_group, hg = h - gi * p.heads_per_group;
    RopeGroup grp = p.group[0];   // selected without indexing the parameter block dynamically
    if (gi == 1) grp = p.group[1];
    if (gi == 2) grp = p.group[2];
    if (gi == 3) grp = p.group[3];
    if (gi == 4) grp = p.group[4];
    if (gi == 5) grp = p.group[5];
    const uint8_t* src0 = reinterpret_cast<const uint8_t*>(p.x) + ((int64_t)h * p.xs_h + x8 * 8) * kBytes;
    uint16_t* dst0 = grp.out + (int64_t)hg * grp.os_h + x8 * 8;
    const float2* fr0 = p.freqs + x8 * 4;
    int b = b0, n = n0;
    constexpr int U = 2;
    for (int r0 = 0; r0 < count; r0 += U) {
      uint4 raw[U][kLoads];
      float4 cs[U][2];
      uint16_t* dst[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (r0 + u >= count) break;
        const uint4* src = reinterpret_cast<const uint4*>(src0 + (b * p.xs_b + n * p.xs_n) * kBytes);
#pragma unroll
        for (int x = 0; x < kLoads; ++x) raw[u][x] = src[x];
        dst[u] = dst0 + b * grp.os_b + n * grp.os_n;
        if (grp.rotate) {
          const float4* fr = reinterpret_cast<const float4*>(fr0 + b * p.fs_b + (int64_t)n * (p.D / 2));
          cs[u][0] = __ldg(fr);
          cs[u][1] = __ldg(fr + 1);
        }
        if constexpr (kSide) {
          b += p.step_b;
          if ((n += p.step_n) >= p.N) n -= p.N, ++b;
        } else if (++n == p.N) {
          n = 0, ++b;
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (r0 + u >= count) break;
        float f[8];
        if constexpr (X_DTYPE == 2) {
          const uint32_t w[8] = {raw[u][0].x, raw[u][0].y, raw[u][0].z, raw[u][0].w, raw[u][kLoads - 1].x,
                                 raw[u][kLoads - 1].y, raw[u][kLoads - 1].z, raw[u][kLoads - 1].w};
#pragma unroll
          for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(w[e]);
        } else {
          constexpr bool kFp16 = X_DTYPE == 1;
          unpack2<kFp16>(raw[u][0].x, f[0], f[1]);
          unpack2<kFp16>(raw[u][0].y, f[2], f[3]);
          unpack2<kFp16>(raw[u][0].z, f[4], f[5]);
          unpack2<kFp16>(raw[u][0].w, f[6], f[7]);
        }
        if (grp.rotate) {
          const float c[8] = {cs[u][0].x, cs[u][0].y, cs[u][0].z, cs[u][0].w, cs[u][1].x, cs[u][1].y, cs[u][1].z, cs[u][1].w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float a = f[2 * i], bb = f[2 * i + 1];
            // (a + bi)(c + si), products and sums rounded separately like the complex multiply
            f[2 * i] = __fsub_rn(__fmul_rn(a, c[2 * i]), __fmul_rn(bb, c[2 * i + 1]));
            f[2 * i + 1] = __fadd_rn(__fmul_rn(a, c[2 * i + 1]), __fmul_rn(bb, c[2 * i]));
          }
        }
        uint4 o;
        if (p.out_fp16) {
          o.x = pack2<true>(f[0], f[1]); o.y = pack2<true>(f[2], f[3]);
          o.z = pack2<true>(f[4], f[5]); o.w = pack2<true>(f[6], f[7]);
        } else {
          o.x = pack2<false>(f[0], f[1]); o.y = pack2<false>(f[2], f[3]);
          o.z = pack2<false>(f[4], f[5]); o.w = pack2<false>(f[6], f[7]);
        }
        *reinterpret_cast<uint4*>(dst[u]) = o;
      }
    }
  }
}

}  // namespace spsattn
