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

// Both gradients in one pass over g: with the window g[t] .. g[t+K-1] in registers, dx[t] is its product with the taps and
// x[t] times the window is what x[t] adds to dw (dw[j] = sum_t x[t] * g[t+(K-1)-j]).  A warp takes 32 channel vectors of one
// run; the CTA adds up its warps' dw and leaves partial[(b * gridDim.y + blockIdx.y), j, c].
// B=8, T=4096, C=4096, 4 taps (0.81 GB): 166 us, 4.9 TB/s, bound by the loads that 12 warps per SM (153 registers) keep in
// flight; two kernels, one per gradient, took 98 + 100 us, 4 channels per thread 197 us, 128 steps per thread 185 us.
template <int KT, bool DX, bool DW>
__global__ void __launch_bounds__(kConvThreads) causal_conv1d_bwd_kernel(const __nv_bfloat16* __restrict__ x,
                                                                         const __nv_bfloat16* __restrict__ w,
                                                                         const __nv_bfloat16* __restrict__ g,
                                                                         __nv_bfloat16* __restrict__ dx, float* __restrict__ partial,
                                                                         int T, int C) {
  constexpr int NB = 4, CW = kConvBwdChannels;
  __shared__ __align__(16) float s_dw[DW ? kConvBwdRuns : 1][DW ? KT : 1][DW ? CW : 4];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c0 = (blockIdx.x * kWarp + lane) * 8, b = blockIdx.z;
  const bool live = c0 < C;
  const int t0 = (blockIdx.y * kConvBwdRuns + warp) * kConvRun, t_end = live ? min(t0 + kConvRun, T) : 0;
  ConvTaps<KT> taps;
  if (DX && live) conv_load_taps<KT>(taps, w, C, c0);
  const long long base = (long long)b * T * C + c0;
  float win[KT][8], acc_w[KT][8];
#pragma unroll
  for (int j = 0; j < KT; ++j)
#pragma unroll
    for (int q = 0; q < 8; ++q) acc_w[j][q] = 0.f;
  if (t0 < t_end) {
#pragma unroll
    for (int i = 0; i < KT - 1; ++i) Elem<__nv_bfloat16>::unpack(conv_fetch(g + base, t0 + i, T, C), win[i]);
  }
  for (int tb = t0; tb < t_end; tb += NB) {
    uint4 raw_g[NB], raw_x[NB];
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      raw_g[i] = conv_fetch(g + base, tb + i + KT - 1, T, C);
      if constexpr (DW) raw_x[i] = conv_fetch(x + base, tb + i, t_end, C);
    }
    const bool tail = tb + NB + KT - 1 > T;   // an x whose g lies past the end adds nothing, also where it is not finite
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      Elem<__nv_bfloat16>::unpack(raw_g[i], win[KT - 1]);
      if constexpr (DX) {
        float acc[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] = 0.f;
#pragma unroll
        for (int j = 0; j < KT; ++j)
#pragma unroll
          for (int q = 0; q < 8; ++q) acc[q] = fmaf(taps.w[KT - 1 - j][q], win[j][q], acc[q]);
        if (tb + i < t_end) st_v4(dx + base + (long long)(tb + i) * C, Elem<__nv_bfloat16>::pack(acc));
      }
      if constexpr (DW) {
        float xv[8];
        Elem<__nv_bfloat16>::unpack(raw_x[i], xv);
#pragma unroll
        for (int j = 0; j < KT; ++j)
          if (!tail || tb + i + KT - 1 - j < T) {
#pragma unroll
            for (int q = 0; q < 8; ++q) acc_w[j][q] = fmaf(xv[q], win[KT - 1 - j][q], acc_w[j][q]);
          }
      }
#pragma unroll
      for (int j = 0; j < KT - 1; ++j)
#pragma unroll
        for (int q = 0; q < 8; ++q) win[j][q] = win[j + 1][q];
    }
  }
  if constexpr (DW) {
#pragma unroll
    for (int j = 0; j < KT; ++j) {
      *reinterpret_cast<float4*>(&s_dw[warp][j][lane * 8]) = make_float4(acc_w[j][0], acc_w[j][1], acc_w[j][2], acc_w[j][3]);
      *reinterpret_cast<float4*>(&s_dw[warp][j][lane * 8 + 4]) = make_float4(acc_w[j][4], acc_w[j][5], acc_w[j][6], acc_w[j][7]);
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
