// Sequence-mixing helpers of the Gated-DeltaNet block that sits beside the MoE layer in the reference's decoder.
// Causal depthwise 1-D convolution (the reference replaces flax's `nnx.Conv(padding="CAUSAL", groups=C)` by K
// shifted multiply-adds, modal/fast_conv.py:14-31):
//   y[b,t,c] = sum_{j<K} w[j,c] * x[b, t-(K-1)+j, c]          (x before the start of the sequence is zero)
// and its gradients
//   dx[b,t,c] = sum_{j<K} w[j,c] * g[b, t+(K-1)-j, c]          (g past the end of the sequence is zero)
//   dw[j,c]   = sum_{b,t} g[b,t,c] * x[b, t-(K-1)+j, c].
// Pure HBM streaming: a thread owns 8 channels (16 bytes) of a run of consecutive time steps and slides a window of
// K vectors through registers, so x is read once (plus K-1 halo steps per run) and y written once.  Products and
// sums are float32, rounded to bf16 once at the end.  The vectors of several time steps are requested before the first
// is used (kConvBatch): the loads in flight are what the bandwidth depends on.
#pragma once

#include "common.cuh"
#include "gather.cuh"
#include "tcgen05.cuh"

namespace lewi {

constexpr int kConvMaxTaps = 8;
constexpr int kConvRun = 32;      // time steps per thread
constexpr int kConvThreads = 128;
constexpr int kConvBwdRuns = kConvThreads / kWarp;   // runs per CTA of the backward kernel, one per warp
constexpr int kConvBwdChannels = kWarp * 8;          // and its channels
template <int KT> constexpr int kConvBatch = KT <= 4 ? 8 : 4;   // time steps requested together (registers)

// KT = number of taps, a compile-time constant so that the sliding window lives in registers.
template <int KT>
struct ConvTaps {
  float w[KT][8];
};

template <int KT>
__device__ __forceinline__ void conv_load_taps(ConvTaps<KT>& taps, const __nv_bfloat16* __restrict__ w, int C, int c0) {
  constexpr int K = KT;
#pragma unroll
  for (int j = 0; j < KT; ++j) {
    if (j < K) {
      float f[8];
      Elem<__nv_bfloat16>::unpack(ld_nc_v4(w + (long long)j * C + c0), f);
#pragma unroll
      for (int q = 0; q < 8; ++q) taps.w[j][q] = f[q];
    }
  }
}

__device__ __forceinline__ uint4 conv_fetch(const __nv_bfloat16* __restrict__ p, int t, int t_end, int C) {
  return t >= 0 && t < t_end ? ld_nc_v4(p + (long long)t * C) : make_uint4(0, 0, 0, 0);
}

// B=8, T=4096, C=4096, 4 taps (0.54 GB): 88 us, 6.1 TB/s (105 us with one vector requested at a time).  NB = kConvBatch<KT>, or 1 for
// one or two steps, since the rest of a batch is worked through for nothing (1024 channels, 4 taps, a batch of 8 and of 1: one
// step 2.0 and 1.7 us, two 2.1 and 1.8, four 2.2 and 2.1, seven 2.3 and 2.5; 8 taps, four 2.2 and 2.6).
template <int KT, int NB>
__global__ void __launch_bounds__(kConvThreads) causal_conv1d_kernel(const __nv_bfloat16* __restrict__ x,
                                                                     const __nv_bfloat16* __restrict__ w,
                                                                     __nv_bfloat16* __restrict__ y, int B, int T, int C) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;      // channel vector
  if (v >= C / 8) return;
  const int c0 = v * 8, b = blockIdx.z, t0 = blockIdx.y * kConvRun, t_end = min(t0 + kConvRun, T);
  ConvTaps<KT> taps;
  conv_load_taps<KT>(taps, w, C, c0);
  const __nv_bfloat16* xb = x + (long long)b * T * C + c0;
  __nv_bfloat16* yb = y + (long long)b * T * C + c0;
  float win[KT][8];   // x[t-(K-1)] .. x[t]
#pragma unroll
  for (int i = 0; i < KT - 1; ++i) Elem<__nv_bfloat16>::unpack(conv_fetch(xb, t0 - (KT - 1) + i, T, C), win[i]);
  for (int tb = t0; tb < t_end; tb += NB) {
    uint4 raw[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) raw[i] = conv_fetch(xb, tb + i, t_end, C);
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      Elem<__nv_bfloat16>::unpack(raw[i], win[KT - 1]);
      float acc[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) acc[q] = 0.f;
#pragma unroll
      for (int j = 0; j < KT; ++j)
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] = fmaf(taps.w[j][q], win[j][q], acc[q]);
      if (tb + i < t_end) st_v4(yb + (long long)(tb + i) * C, Elem<__nv_bfloat16>::pack(acc));
#pragma unroll
      for (int j = 0; j < KT - 1; ++j)
#pragma unroll
        for (int q = 0; q < 8; ++q) win[j][q] = win[j + 1][q];
    }
  }
}

// Two floats side by side (fma.rn.f32x2: each half rounded as a single fma).
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 f2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void f2_split(F2 a, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(a.v)); }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ void unpack2(uint4 v, F2 (&f)[4]) {
  f[0] = f2(bf16_lo(v.x), bf16_hi(v.x));
  f[1] = f2(bf16_lo(v.y), bf16_hi(v.y));
  f[2] = f2(bf16_lo(v.z), bf16_hi(v.z));
  f[3] = f2(bf16_lo(v.w), bf16_hi(v.w));
}
__device__ __forceinline__ uint32_t f2_bf16(F2 a) {
  float lo, hi;
  f2_split(a, lo, hi);
  return pack_bf16(lo, hi);
}

// Both gradients in one pass over g: with the window g[t] .. g[t+K-1] in registers, dx[t] is its product with the taps and
// x[t] times the window is what x[t] adds to dw (dw[j] = sum_t x[t] * g[t+(K-1)-j]).  A warp takes 32 channel vectors of one
// run; the CTA adds up its warps' dw and leaves partial[(b * gridDim.y + blockIdx.y), j, c].
// What bounds it are the loads in flight: a lane's vectors go through a ring of its own in shared memory (cp.async; no other lane reads
// them, so nothing is synchronised), kConvBwdStages batches of kConvBwdBatch steps deep, and channels are worked through in pairs.
// B=8, T=4096, C=4096, 4 taps (0.81 GB): 132 us, 6.1 TB/s; with the batches in registers 166 us, 4.9 TB/s; two kernels, one per
// gradient, took 98 + 100 us, 4 channels per thread 197 us, 128 steps per thread 185 us.
constexpr int kConvBwdBatch = 4, kConvBwdStages = 3;
template <bool DW> constexpr int conv_bwd_ring() { return kConvThreads * kConvBwdStages * kConvBwdBatch * (DW ? 2 : 1) * 16; }
template <int KT, bool DX, bool DW>
__global__ void __launch_bounds__(kConvThreads) causal_conv1d_bwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                                         const __nv_bfloat16* __restrict__ w,
                                                                         const __nv_bfloat16* __restrict__ g,
                                                                         __nv_bfloat16* __restrict__ dx, float* __restrict__ partial,
                                                                         int T, int C) {
  constexpr int NB = kConvBwdBatch, ST = kConvBwdStages, CW = kConvBwdChannels, VEC = DW ? 2 : 1;
  extern __shared__ __align__(16) uint8_t conv_ring[];   // [stage][step][g, x][thread] vectors; at the end the warps' dw
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c0 = (blockIdx.x * kWarp + lane) * 8, b = blockIdx.z;
  const bool live = c0 < C;
  const int t0 = (blockIdx.y * kConvBwdRuns + warp) * kConvRun, t_end = live ? min(t0 + kConvRun, T) : 0;
  F2 taps[KT][4];
  if (DX && live) {
#pragma unroll
    for (int j = 0; j < KT; ++j) unpack2(ld_nc_v4(w + (long long)j * C + c0), taps[j]);
  }
  const long long base = (long long)b * T * C + c0;
  const uint4* mine = reinterpret_cast<const uint4*>(conv_ring) + threadIdx.x;
  const uint32_t mine_at = ptx::smem_u32(mine);
  auto fetch = [&](int batch) {   // (always a group, also an empty one, so that the groups count the batches)
    const int tb = t0 + batch * NB, slot = batch % ST * NB * VEC;
    if (tb < t_end) {
#pragma unroll
      for (int i = 0; i < NB; ++i) {
        const int tg = tb + i + KT - 1;
        ptx::cp_async16(mine_at + (slot + i * VEC) * (kConvThreads * 16), g + base + (long long)min(tg, T - 1) * C, tg < T ? 16u : 0u);
        if constexpr (DW)
          ptx::cp_async16(mine_at + (slot + i * VEC + 1) * (kConvThreads * 16), x + base + (long long)min(tb + i, T - 1) * C,
                          tb + i < t_end ? 16u : 0u);
      }
    }
    ptx::cp_async_commit();
  };
  F2 win[KT][4], acc_w[KT][4];
#pragma unroll
  for (int j = 0; j < KT; ++j)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc_w[j][q] = f2(0.f, 0.f);
#pragma unroll
  for (int s = 0; s < ST; ++s) fetch(s);
  if (t0 < t_end) {
#pragma unroll
    for (int i = 0; i < KT - 1; ++i) unpack2(conv_fetch(g + base, t0 + i, T, C), win[i]);
  }
  for (int tb = t0, batch = 0; tb < t_end; tb += NB, ++batch) {
    ptx::cp_async_wait<ST - 1>();
    const int slot = batch % ST * NB * VEC;
    const bool tail = tb + NB + KT - 1 > T;   // an x whose g lies past the end adds nothing, also where it is not finite
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      unpack2(mine[(slot + i * VEC) * kConvThreads], win[KT - 1]);
      if constexpr (DX) {
        F2 acc[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] = f2(0.f, 0.f);
#pragma unroll
        for (int j = 0; j < KT; ++j)
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[q] = fma2(taps[KT - 1 - j][q], win[j][q], acc[q]);
        if (tb + i < t_end) st_v4(dx + base + (long long)(tb + i) * C, make_uint4(f2_bf16(acc[0]), f2_bf16(acc[1]), f2_bf16(acc[2]), f2_bf16(acc[3])));
      }
      if constexpr (DW) {
        F2 xv[4];
        unpack2(mine[(slot + i * VEC + 1) * kConvThreads], xv);
#pragma unroll
        for (int j = 0; j < KT; ++j)
          if (!tail || tb + i + KT - 1 - j < T) {
#pragma unroll
            for (int q = 0; q < 4; ++q) acc_w[j][q] = fma2(xv[q], win[KT - 1 - j][q], acc_w[j][q]);
          }
      }
#pragma unroll
      for (int j = 0; j < KT - 1; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) win[j][q] = win[j + 1][q];
    }
    fetch(batch + ST);   // (the batch just worked through has left the ring)
  }
  ptx::cp_async_wait<0>();
  if constexpr (DW) {
    float (*s_dw)[KT][CW] = reinterpret_cast<float (*)[KT][CW]>(conv_ring);
    __syncthreads();   // the other warps' vectors have been read
#pragma unroll
    for (int j = 0; j < KT; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float lo, hi;
        f2_split(acc_w[j][q], lo, hi);
        *reinterpret_cast<float2*>(&s_dw[warp][j][lane * 8 + 2 * q]) = make_float2(lo, hi);
      }
    __syncthreads();
    float* dst = partial + ((long long)b * gridDim.y + blockIdx.y) * KT * C;
    for (int i = threadIdx.x; i < KT * CW / 4; i += kConvThreads) {
      const int j = i / (CW / 4), cc = i % (CW / 4) * 4, c = blockIdx.x * CW + cc;
      if (c >= C) continue;
      float4 sum = *reinterpret_cast<const float4*>(&s_dw[0][j][cc]);
#pragma unroll
      for (int r = 1; r < kConvBwdRuns; ++r) {
        const float4 p = *reinterpret_cast<const float4*>(&s_dw[r][j][cc]);
        sum.x += p.x; sum.y += p.y; sum.z += p.z; sum.w += p.w;
      }
      *reinterpret_cast<float4*>(dst + (long long)j * C + c) = sum;
    }
  }
}

template <int KT, bool DX, bool DW>
inline int launch_conv_bwd(dim3 grid, cudaStream_t st, const __nv_bfloat16* x, const __nv_bfloat16* w, const __nv_bfloat16* g,
                           __nv_bfloat16* dx, float* partial, int T, int C) {
  static bool done[64] = {false};
  constexpr int ring = conv_bwd_ring<DW>(), sums = DW ? kConvBwdRuns * KT * kConvBwdChannels * 4 : 0, smem = ring > sums ? ring : sums;
  if (!allow_smem(causal_conv1d_bwd_kernel<KT, DX, DW>, smem, done)) return LEWI_ERR_CUDA;
  causal_conv1d_bwd_kernel<KT, DX, DW><<<grid, kConvThreads, smem, st>>>(x, w, g, dx, partial, T, C);
  return LEWI_OK;
}

// out[i] = sum over parts of partial[part, i], n a multiple of 4: a CTA takes 32 vectors of 4 columns, its warps every 8th part
// each; sums in a fixed order.  (One thread per column walked all parts: 61 us for 1024 parts of 16384 columns; now 10 us for 256.)
__global__ void __launch_bounds__(256) conv_dw_reduce_kernel(const float* __restrict__ partial, int n_parts, int n,
                                                             __nv_bfloat16* __restrict__ out_bf16, float* __restrict__ out_f32) {
  __shared__ float4 s_sum[8][kWarp];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int i = (blockIdx.x * kWarp + lane) * 4;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  if (i < n) {
#pragma unroll 8
    for (int p = warp; p < n_parts; p += 8) {
      const float4 v = *reinterpret_cast<const float4*>(partial + (long long)p * n + i);
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
  }
  s_sum[warp][lane] = acc;
  __syncthreads();
  if (warp != 0 || i >= n) return;
#pragma unroll
  for (int r = 1; r < 8; ++r) {
    const float4 v = s_sum[r][lane];
    acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
  }
  const float o[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {   // (the output need not be aligned)
    if (out_f32 != nullptr) out_f32[i + q] = o[q];
    if (out_bf16 != nullptr) out_bf16[i + q] = __float2bfloat16_rn(o[q]);
  }
}

}  // namespace lewi
