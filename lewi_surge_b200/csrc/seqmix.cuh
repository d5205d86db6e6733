// Sequence-mixing helpers of the Gated-DeltaNet block that sits beside the MoE layer in the reference's decoder.
// Causal depthwise 1-D convolution (the reference replaces flax's `nnx.Conv(padding="CAUSAL", groups=C)` by K
// shifted multiply-adds, modal/fast_conv.py:14-31):
//   y[b,t,c] = sum_{j<K} w[j,c] * x[b, t-(K-1)+j, c]          (x before the start of the sequence is zero)
// and its gradients
//   dx[b,t,c] = sum_{j<K} w[j,c] * g[b, t+(K-1)-j, c]          (g past the end of the sequence is zero)
//   dw[j,c]   = sum_{b,t} g[b,t,c] * x[b, t-(K-1)+j, c].
// Pure HBM streaming: a thread owns 8 channels (16 bytes) of a run of consecutive time steps and slides a window of
// K vectors through registers, so x is read once (plus K-1 halo steps per run) and y written once.  Products and
// sums are float32, rounded to bf16 once at the end.
#pragma once

#include "common.cuh"
#include "gather.cuh"

namespace lewi {

constexpr int kConvMaxTaps = 8;
constexpr int kConvRun = 32;      // time steps per thread
constexpr int kConvThreads = 128;

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

// REVERSE = false: forward (window looks back in time); true: the input gradient (window looks ahead, taps flipped).
template <bool REVERSE, int KT>
__global__ void __launch_bounds__(kConvThreads) causal_conv1d_kernel(const __nv_bfloat16* __restrict__ x,
                                                                     const __nv_bfloat16* __restrict__ w,
                                                                     __nv_bfloat16* __restrict__ y, int B, int T, int C) {
  constexpr int K = KT;
  const int cvec = C / 8;
  const int v = blockIdx.x * blockDim.x + threadIdx.x;      // channel vector
  if (v >= cvec) return;
  const int c0 = v * 8;
  const int run = blockIdx.y, b = blockIdx.z;
  const int t0 = run * kConvRun;
  ConvTaps<KT> taps;
  conv_load_taps<KT>(taps, w, C, c0);
  const __nv_bfloat16* xb = x + (long long)b * T * C + c0;
  __nv_bfloat16* yb = y + (long long)b * T * C + c0;
  float win[KT][8];   // win[i] = input at offset i of the current window
  auto fetch = [&](int t, float* dst) {
    if (t >= 0 && t < T) {
      Elem<__nv_bfloat16>::unpack(ld_nc_v4(xb + (long long)t * C), dst);
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) dst[q] = 0.f;
    }
  };
  // forward: output t reads inputs t-(K-1) .. t, tap j at window slot j
  // reverse: output t reads inputs t .. t+(K-1), input t+i meets tap K-1-i
#pragma unroll
  for (int i = 0; i < KT; ++i)
    if (i < K - 1) fetch(REVERSE ? t0 + i : t0 - (K - 1) + i, win[i]);
  const int t_end = min(t0 + kConvRun, T);
  for (int t = t0; t < t_end; ++t) {
    fetch(REVERSE ? t + (K - 1) : t, win[K - 1]);
    float acc[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] = 0.f;
#pragma unroll
    for (int i = 0; i < KT; ++i) {
      if (i < K) {
        const int j = REVERSE ? K - 1 - i : i;
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] = fmaf(taps.w[j][q], win[i][q], acc[q]);
      }
    }
    st_v4(yb + (long long)t * C, Elem<__nv_bfloat16>::pack(acc));
#pragma unroll
    for (int i = 0; i < KT - 1; ++i)
      if (i < K - 1) {
#pragma unroll
        for (int q = 0; q < 8; ++q) win[i][q] = win[i + 1][q];
      }
  }
}

// partial[(b * runs + run), j, c] = sum over the run's time steps of g[b,t,c] * x[b, t-(K-1)+j, c]
template <int KT>
__global__ void __launch_bounds__(kConvThreads) causal_conv1d_dw_kernel(const __nv_bfloat16* __restrict__ x,
                                                                        const __nv_bfloat16* __restrict__ g,
                                                                        float* __restrict__ partial, int B, int T, int C) {
  constexpr int K = KT;
  const int cvec = C / 8;
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= cvec) return;
  const int c0 = v * 8;
  const int run = blockIdx.y, b = blockIdx.z;
  const int t0 = run * kConvRun;
  const __nv_bfloat16* xb = x + (long long)b * T * C + c0;
  const __nv_bfloat16* gb = g + (long long)b * T * C + c0;
  float win[KT][8], acc[KT][8];
#pragma unroll
  for (int j = 0; j < KT; ++j)
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[j][q] = 0.f;
  auto fetch = [&](int t, float* dst) {
    if (t >= 0 && t < T) {
      Elem<__nv_bfloat16>::unpack(ld_nc_v4(xb + (long long)t * C), dst);
    } else {
#pragma unroll
      for (int q = 0; q < 8; ++q) dst[q] = 0.f;
    }
  };
#pragma unroll
  for (int i = 0; i < KT; ++i)
    if (i < K - 1) fetch(t0 - (K - 1) + i, win[i]);
  const int t_end = min(t0 + kConvRun, T);
  for (int t = t0; t < t_end; ++t) {
    fetch(t, win[K - 1]);
    float gv[8];
    Elem<__nv_bfloat16>::unpack(ld_nc_v4(gb + (long long)t * C), gv);
#pragma unroll
    for (int j = 0; j < KT; ++j)
      if (j < K) {
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[j][q] = fmaf(gv[q], win[j][q], acc[j][q]);
      }
#pragma unroll
    for (int i = 0; i < KT - 1; ++i)
      if (i < K - 1) {
#pragma unroll
        for (int q = 0; q < 8; ++q) win[i][q] = win[i + 1][q];
      }
  }
  const long long part = (long long)b * gridDim.y + run;
#pragma unroll
  for (int j = 0; j < KT; ++j)
    if (j < K) {
      float* dst = partial + (part * K + j) * C + c0;
      *reinterpret_cast<float4*>(dst) = make_float4(acc[j][0], acc[j][1], acc[j][2], acc[j][3]);
      *reinterpret_cast<float4*>(dst + 4) = make_float4(acc[j][4], acc[j][5], acc[j][6], acc[j][7]);
    }
}

// out[i] (bf16) = sum over parts of partial[part, i]; the parts of a column are added in index order.
__global__ void __launch_bounds__(256) conv_dw_reduce_kernel(const float* __restrict__ partial, int n_parts, int n,
                                                             __nv_bfloat16* __restrict__ out_bf16, float* __restrict__ out_f32) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float acc = 0.f;
  for (int p = 0; p < n_parts; ++p) acc += partial[(long long)p * n + i];
  if (out_f32 != nullptr) out_f32[i] = acc;
  if (out_bf16 != nullptr) out_bf16[i] = __float2bfloat16_rn(acc);
}

}  // namespace lewi
