// Element-wise kernels that sit between the attention calls and the projections of an SPS
// decoder block, so that a generation step is a short fixed chain of launches: residual add +
// RMSNorm in one pass, and the SwiGLU gate.  Both are bandwidth bound and keep the reference's
// rounding points for 16-bit parameters (every torch op there rounds its result to bf16).
// Reference computation: RMSNorm src/modeling/models/model.py:101-132 (normalise in fp32, cast
// back to the input type, then multiply by the weight), residual adds :324-327, MLP :304-314
// (down(silu(gate(x)) * up(x))).
#pragma once

#include "common.cuh"

namespace spsattn {

struct RmsNormParams {
  void* x;             // [rows, C] residual stream, updated in place when delta is given
  const void* delta;   // [rows, C] or null
  const void* weight;  // [C]
  void* y;             // [rows, C] normalised output
  long long rows;
  int C;
  float eps;
  int let_go;          // when dependents may start (they wait themselves before they read y): NormLetGo
};

// At once only inside a decode step: what dependents touch before their own wait (weights, rows of a cache), and
// this kernel's own weight, is then no longer being written by anything.  After the wait: where a step's launches begin
// and what stands before them is not known, as in token_start_kernel.
enum NormLetGo { kLetGoAtEnd = 0, kLetGoAtOnce = 1, kLetGoAfterWait = 2 };

__device__ __forceinline__ float round_bf16(float f) {
  return __bfloat162float(__float2bfloat16_rn(f));
}

// One block per row.  BF16 = true: x, delta, weight, y are bf16 and results are rounded where the
// reference's bf16 tensors round; false: everything fp32.  A row of up to 256 * kRowVecs vectors
// stays in registers between the sum of squares and the scaling (one read of x); longer rows are
// read again.
// kAhead: a block has its next row on the way while it works on this one.  That takes registers (with
// kRowVecs 1 six blocks per SM still fit, 174 us against 202 with five; with 4 only two), which wide rows
// need for more blocks: without it 65536 bf16 rows of 4096 357 -> 260 us, 16384 fp32 rows of 8192 310 -> 177.
// kStep: inside a decode step, rows of at most 256 vectors; the few blocks have registers to keep the weight.
template <bool BF16, int kRowVecs, bool kAhead, bool kStep = false>
__global__ void __launch_bounds__(256, kStep ? 2 : kRowVecs == 1 ? 6 : kAhead ? 2 : 4) add_rmsnorm_kernel(const RmsNormParams p) {
  constexpr int V = BF16 ? 8 : 4;   // elements per 16-byte access
  __shared__ float s_part[2][8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n_vec = p.C / V;
  const bool in_regs = n_vec <= 256 * kRowVecs;
  uint4* const px = reinterpret_cast<uint4*>(p.x);
  const uint4* const pd = reinterpret_cast<const uint4*>(p.delta);
  const uint4* const pw = reinterpret_cast<const uint4*>(p.weight);
  uint4* const py = reinterpret_cast<uint4*>(p.y);

  auto unpack = [](const uint4& u, float (&f)[V]) {
    if constexpr (BF16) {
      unpack2<false>(u.x, f[0], f[1]);
      unpack2<false>(u.y, f[2], f[3]);
      unpack2<false>(u.z, f[4], f[5]);
      unpack2<false>(u.w, f[6], f[7]);
    } else {
      f[0] = __uint_as_float(u.x), f[1] = __uint_as_float(u.y), f[2] = __uint_as_float(u.z), f[3] = __uint_as_float(u.w);
    }
  };
  auto pack = [](const float (&f)[V]) {
    if constexpr (BF16)
      return make_uint4(pack2<false>(f[0], f[1]), pack2<false>(f[2], f[3]), pack2<false>(f[4], f[5]), pack2<false>(f[6], f[7]));
    else
      return make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
  };
  // x + delta of one vector (written back), or x
  auto sum = [&](size_t at, const uint4& u, const uint4& d, float (&f)[V]) {
    unpack(u, f);
    if (p.delta != nullptr) {
      float g[V];
      unpack(d, g);
#pragma unroll
      for (int e = 0; e < V; ++e) f[e] = BF16 ? round_bf16(f[e] + g[e]) : f[e] + g[e];
      px[at] = pack(f);
    }
  };
  // kStep: the weight is read before the wait, not behind the barrier (us per token: 12 layers of 1024 columns, 32 rows
  // 395 -> 379; 12 x 768, 18 rows 345 -> 339; 4 x 2048, 32 rows 337 -> 332).
  uint4 wgt = make_uint4(0, 0, 0, 0);
  auto store_y = [&](size_t at, int i, const float (&f)[V], float scale) {
    float g[V], r[V];
    unpack(kStep ? wgt : __ldg(pw + i), g);
#pragma unroll
    for (int e = 0; e < V; ++e) r[e] = BF16 ? round_bf16(f[e] * scale) * g[e] : f[e] * scale * g[e];
    py[at] = pack(r);
  };

  // Bound: HBM.  A block synchronises once per row (every thread adds the eight warp sums itself, in the
  // same order): 65536 rows of 2048 with delta 250 -> 174 us, 6.2 TB/s.
  if (p.let_go != kLetGoAtOnce) grid_dependency_wait();
  if (p.let_go != kLetGoAtEnd) grid_launch_dependents();
  if (kStep && tid < n_vec) wgt = __ldg(pw + tid);
  if (p.let_go == kLetGoAtOnce) grid_dependency_wait();
  uint4 nx[kRowVecs], nd[kRowVecs];
  auto fetch = [&](long long row) {
    if (!in_regs || row >= p.rows) return;
#pragma unroll
    for (int k = 0; k < kRowVecs; ++k) {
      const int i = tid + k * 256;
      if (i < n_vec) {
        nx[k] = px[(size_t)row * n_vec + i];
        if (p.delta != nullptr) nd[k] = pd[(size_t)row * n_vec + i];
      }
    }
  };
  if constexpr (kAhead) fetch(blockIdx.x);
  int buf = 0;
  for (long long row = blockIdx.x; row < p.rows; row += gridDim.x, buf ^= 1) {
    const size_t base = (size_t)row * n_vec;
    float ss = 0.f;
    float kept[kRowVecs][V];
    if (in_regs) {
#pragma unroll
      for (int k = 0; k < kRowVecs; ++k) {
        const int i = tid + k * 256;
        if (i < n_vec) {
          if constexpr (kAhead) sum(base + i, nx[k], nd[k], kept[k]);
          else sum(base + i, px[base + i], p.delta != nullptr ? pd[base + i] : make_uint4(0, 0, 0, 0), kept[k]);
#pragma unroll
          for (int e = 0; e < V; ++e) ss = fmaf(kept[k][e], kept[k][e], ss);
        }
      }
      if constexpr (kAhead) fetch(row + gridDim.x);
    } else {
      for (int i = tid; i < n_vec; i += 256) {
        float f[V];
        sum(base + i, px[base + i], p.delta != nullptr ? pd[base + i] : make_uint4(0, 0, 0, 0), f);
#pragma unroll
        for (int e = 0; e < V; ++e) ss = fmaf(f[e], f[e], ss);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (lane == 0) s_part[buf][warp] = ss;
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += s_part[buf][w];
    const float scale = rsqrtf(t / (float)p.C + p.eps);
    if (p.y != nullptr) {
      if (in_regs) {
#pragma unroll
        for (int k = 0; k < kRowVecs; ++k) {
          const int i = tid + k * 256;
          if (i < n_vec) store_y(base + i, i, kept[k], scale);
        }
      } else {
        // second read: x already holds the sum
        for (int i = tid; i < n_vec; i += 256) {
          float f[V];
          unpack(px[base + i], f);
          store_y(base + i, i, f, scale);
        }
      }
    }
  }
}

struct SwigluParams {
  const void* gate_up;   // [rows, 2 * I]: gate in columns [0, I), up in [I, 2I)
  void* y;               // [rows, I]
  long long rows;
  int I;
};

__device__ __forceinline__ float silu_f(float x) { return x / (1.f + expf(-x)); }

template <bool BF16>
__global__ void __launch_bounds__(256) swiglu_kernel(const SwigluParams p) {
  constexpr int V = BF16 ? 8 : 4;
  grid_dependency_wait();
  const int n_vec = p.I / V;
  const long long total = p.rows * n_vec;
  for (long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x; idx < total;
       idx += (long long)gridDim.x * blockDim.x) {
    const long long row = idx / n_vec;
    const int i = (int)(idx % n_vec);
    const size_t src = (size_t)row * 2 * p.I + (size_t)i * V;
    const size_t dst = (size_t)row * p.I + (size_t)i * V;
    if constexpr (BF16) {
      const uint16_t* gp = reinterpret_cast<const uint16_t*>(p.gate_up);
      const uint4 a = *reinterpret_cast<const uint4*>(gp + src);
      const uint4 b = *reinterpret_cast<const uint4*>(gp + src + p.I);
      float g[8], u[8];
      unpack2<false>(a.x, g[0], g[1]); unpack2<false>(a.y, g[2], g[3]);
      unpack2<false>(a.z, g[4], g[5]); unpack2<false>(a.w, g[6], g[7]);
      unpack2<false>(b.x, u[0], u[1]); unpack2<false>(b.y, u[2], u[3]);
      unpack2<false>(b.z, u[4], u[5]); unpack2<false>(b.w, u[6], u[7]);
#pragma unroll
      for (int e = 0; e < 8; ++e) g[e] = round_bf16(silu_f(g[e])) * u[e];
      uint4 o;
      o.x = pack2<false>(g[0], g[1]); o.y = pack2<false>(g[2], g[3]);
      o.z = pack2<false>(g[4], g[5]); o.w = pack2<false>(g[6], g[7]);
      *reinterpret_cast<uint4*>(reinterpret_cast<uint16_t*>(p.y) + dst) = o;
    } else {
      const float* gp = reinterpret_cast<const float*>(p.gate_up);
      const float4 a = *reinterpret_cast<const float4*>(gp + src);
      const float4 b = *reinterpret_cast<const float4*>(gp + src + p.I);
      *reinterpret_cast<float4*>(reinterpret_cast<float*>(p.y) + dst) =
          make_float4(silu_f(a.x) * b.x, silu_f(a.y) * b.y, silu_f(a.z) * b.z, silu_f(a.w) * b.w);
    }
  }
}

}  // namespace spsattn
