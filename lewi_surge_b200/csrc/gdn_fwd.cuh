// Chunked gated delta rule, forward (the reference's `fast_chunk_gated_delta_rule`, modal/gdn_fast.py:37-113).
//
// Per (batch, head) the state h [K,V] follows  h <- h*exp(g_t) + k_t (x) beta_t (v_t - k_t^T h),  o_t = q_t^T h.
// Tokens are processed in chunks of 64 (WY form): with gcs = cumsum(g) inside the chunk,
//   S    = strict_lower( bf16(k_beta k^T) * exp(gcs_i - gcs_j) ),   A = (I + S)^-1,
//   u    = bf16(A v_beta),   w = bf16(A (k_beta * exp(gcs))),
//   attn = lower( bf16(q k^T) * exp(gcs_i - gcs_j) )
// depend on one chunk only (chunk kernel, one CTA per chunk and head), and the recurrence over chunks
//   v_new = u - w h;   o = (q exp(gcs)) h + attn v_new;   h <- h exp(gcs_last) + (k exp(gcs_last - gcs))^T v_new
// is independent per column of h (scan kernel, one warp per 16 columns of V).  The roundings to bf16 are the ones JAX
// applies in the reference for compute_dtype = bfloat16; everything that involves g or the state is float32, like the
// reference at its default precision: those operands enter the tensor cores in three bf16 pieces (gdn_mma.cuh).
#pragma once

#include "gdn_mma.cuh"
#include "gather.cuh"
#include "grouped_gemm.cuh"

namespace lewi {
namespace gdn {

constexpr int kChunkThreads = 256;
constexpr int kSP = 68;   // row stride (floats) of the [64][64] float32 arrays: 16-byte rows, odd multiple of 4 banks

// The A operand (16 rows from r0, 16 columns from c0) and the B operand (16 rows from k0, 8 columns from n0) of a product of
// float32 matrices in shared memory (row stride kSP), in three pieces.
__device__ __forceinline__ void f32_a(const float* m, int r0, int c0, int lane, Frag3x4& f) {
  const float* p = m + (r0 + (lane >> 2)) * kSP + c0 + (lane & 3) * 2;
  const float2 x0 = *reinterpret_cast<const float2*>(p), x1 = *reinterpret_cast<const float2*>(p + 8 * kSP);
  const float2 x2 = *reinterpret_cast<const float2*>(p + 8), x3 = *reinterpret_cast<const float2*>(p + 8 * kSP + 8);
  split3(x0.x, x0.y, f.p[0][0], f.p[1][0], f.p[2][0]);
  split3(x1.x, x1.y, f.p[0][1], f.p[1][1], f.p[2][1]);
  split3(x2.x, x2.y, f.p[0][2], f.p[1][2], f.p[2][2]);
  split3(x3.x, x3.y, f.p[0][3], f.p[1][3], f.p[2][3]);
}
__device__ __forceinline__ void f32_b(const float* m, int k0, int n0, int lane, uint32_t (&b)[3][2]) {
  const float* p = m + (k0 + (lane & 3) * 2) * kSP + n0 + (lane >> 2);
  split3(p[0], p[kSP], b[0][0], b[1][0], b[2][0]);
  split3(p[8 * kSP], p[9 * kSP], b[0][1], b[1][1], b[2][1]);
}
__device__ __forceinline__ void mma_x6(float (&d)[4], const Frag3x4& a, const uint32_t (&b)[3][2]) {
  float t[4];
  zero4(t);
  mma(t, a.p[0], b[2][0], b[2][1]);
  mma(t, a.p[2], b[0][0], b[0][1]);
  mma(t, a.p[1], b[1][0], b[1][1]);
  mma(t, a.p[0], b[1][0], b[1][1]);
  mma(t, a.p[1], b[0][0], b[0][1]);
  mma(t, a.p[0], b[0][0], b[0][1]);
  add4(d, t);
}

// A = (I + S)^-1 for the strictly lower S in sS; A (lower, exact zeros above the diagonal) goes to sA.  All threads, 256 or more.
// Inverse by halves: the four 16 x 16 diagonal blocks by forward substitution (64 threads, a column each: 15 dependent
// sums instead of the 63 of the whole matrix), then A_lower-left = -A_bottom (S_lower-left A_top) for blocks of 16 and 32 on
// the tensor cores.  sX is scratch of [32][kSP] floats.  Ends with a barrier.  (Whole-matrix substitution took 11,000 cycles.)
__device__ __forceinline__ void unit_lower_inverse(const float* sS, float* sA, float* sX, int tid) {
  const int lane = tid & 31, warp = tid >> 5;
  if (tid < C) {
    const int d0 = tid & ~15, c = tid & 15;
    const float* S = sS + d0 * kSP + d0;
    float col[16];   // stored only at the end: a store in between would hold up the loads of the next row
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      float acc = i == c ? 1.f : 0.f;
#pragma unroll
      for (int j4 = 0; j4 < i; j4 += 4) {
        const float4 s4 = *reinterpret_cast<const float4*>(S + i * kSP + j4);
        acc = fmaf(-s4.x, col[j4], acc);
        if (j4 + 1 < i) acc = fmaf(-s4.y, col[j4 + 1], acc);
        if (j4 + 2 < i) acc = fmaf(-s4.z, col[j4 + 2], acc);
        if (j4 + 3 < i) acc = fmaf(-s4.w, col[j4 + 3], acc);
      }
      col[i] = i < c ? 0.f : acc;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) sA[(d0 + i) * kSP + d0 + c] = col[i];
  } else {   // everything above the diagonal blocks
    for (int i = tid - C; i < C * C / 4; i += (int)blockDim.x - C) {
      const int r = i >> 4, c = (i & 15) * 4;
      if ((c >> 4) > (r >> 4)) *reinterpret_cast<float4*>(sA + r * kSP + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  __syncthreads();
  const int er = lane >> 2, ec = (lane & 3) * 2;   // this lane's elements of an accumulator tile
  // blocks of 16: warps 0-3, pair = warp/2 (rows 32*pair ..), 8 columns each
  if (warp < 4) {
    const int t0 = (warp >> 1) * 32, n0 = (warp & 1) * 8;
    float acc[4];
    Frag3x4 fa;
    uint32_t fb[3][2];
    zero4(acc);
    f32_a(sS, t0 + 16, t0, lane, fa);
    f32_b(sA, t0, t0 + n0, lane, fb);
    mma_x6(acc, fa, fb);
    float* x = sX + (warp >> 1) * 16 * kSP + er * kSP + n0 + ec;
    *reinterpret_cast<float2*>(x) = make_float2(-acc[0], -acc[1]);
    *reinterpret_cast<float2*>(x + 8 * kSP) = make_float2(-acc[2], -acc[3]);
    __syncwarp();
    // the second product needs only this warp's own columns of the first
    zero4(acc);
    f32_a(sA, t0 + 16, t0 + 16, lane, fa);
    f32_b(sX, (warp >> 1) * 16, n0, lane, fb);
    mma_x6(acc, fa, fb);
    float* o = sA + (t0 + 16 + er) * kSP + t0 + n0 + ec;
    *reinterpret_cast<float2*>(o) = make_float2(acc[0], acc[1]);
    *reinterpret_cast<float2*>(o + 8 * kSP) = make_float2(acc[2], acc[3]);
  }
  __syncthreads();
  // blocks of 32: warps 0-7, (16 rows, 8 columns) each
  const int m0 = ((warp & 7) >> 2) * 16, n0 = (warp & 3) * 8;
  float acc[4];
  Frag3x4 fa;
  uint32_t fb[3][2];
  if (warp < 8) {
    zero4(acc);
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      f32_a(sS, 32 + m0, ks * 16, lane, fa);
      f32_b(sA, ks * 16, n0, lane, fb);
      mma_x6(acc, fa, fb);
    }
    float* x = sX + (m0 + er) * kSP + n0 + ec;
    *reinterpret_cast<float2*>(x) = make_float2(-acc[0], -acc[1]);
    *reinterpret_cast<float2*>(x + 8 * kSP) = make_float2(-acc[2], -acc[3]);
  }
  __syncthreads();
  if (warp < 8) {
    zero4(acc);
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
      f32_a(sA, 32 + m0, 32 + ks * 16, lane, fa);
      f32_b(sX, ks * 16, n0, lane, fb);
      mma_x6(acc, fa, fb);
    }
    float* o = sA + (32 + m0 + er) * kSP + n0 + ec;
    *reinterpret_cast<float2*>(o) = make_float2(acc[0], acc[1]);
    *reinterpret_cast<float2*>(o + 8 * kSP) = make_float2(acc[2], acc[3]);
  }
  __syncthreads();
}

// Prefix sums of g and the decay factors of one chunk by warp 0: gates[0] = gcs, [1] = exp(gcs), [2] = exp(gcs_last - gcs).
// The sum runs over the tokens in order, in every lane: the decay between two tokens is then off by the roundings between them
// only.  (Prefixes by shuffles, each with roundings of its own, left the in-chunk attention 1.5 times as far from 64 bits.)
__device__ __forceinline__ void chunk_gates(float* gates, float g0, float g1, int lane) {   // g of tokens 2*lane, 2*lane+1
  *reinterpret_cast<float2*>(gates + 2 * lane) = make_float2(g0, g1);
  __syncwarp();
  float last = 0.f, a = 0.f, b = 0.f;
#pragma unroll
  for (int i = 0; i < C / 4; ++i) {
    const float4 x = *reinterpret_cast<const float4*>(gates + 4 * i);
    last += x.x;
    a = 2 * i == lane ? last : a;
    last += x.y;
    b = 2 * i == lane ? last : b;
    last += x.z;
    a = 2 * i + 1 == lane ? last : a;
    last += x.w;
    b = 2 * i + 1 == lane ? last : b;
  }
  __syncwarp();
  gates[2 * lane] = a;
  gates[2 * lane + 1] = b;
  gates[C + 2 * lane] = __expf(a);
  gates[C + 2 * lane + 1] = __expf(b);
  gates[2 * C + 2 * lane] = __expf(last - a);
  gates[2 * C + 2 * lane + 1] = __expf(last - b);
}

// ------------------------------------------------------------------------------------------------ chunk kernel

// Shared memory of the chunk kernel: tiles k, q*scale and k*beta (KB boxes each; k and q later hold the pieces of A), v*beta
// (128 columns at a time), the pieces of A exp(gcs), S and A in float32, scratch of the inverse, gates.
struct ChunkSmem {
  int k, q, kb, v, pa, pae, s, a, x, gates, total;
};
__host__ __device__ constexpr ChunkSmem chunk_smem(int kboxes) {
  ChunkSmem m{};
  m.k = 0;
  m.q = kboxes * kBox;
  m.pa = 0;                                       // three boxes over k and q once those have been used
  m.kb = kboxes == 1 ? 3 * kBox : 2 * kboxes * kBox;
  m.v = m.kb + kboxes * kBox;
  m.pae = m.v + 2 * kBox;
  m.s = m.pae;                                    // S and the scratch are dead before the pieces of A exp(gcs) are made
  m.x = m.s + C * kSP * 4;
  m.a = m.x + 32 * kSP * 4;
  if (m.a < m.pae + 3 * kBox) m.a = m.pae + 3 * kBox;
  m.gates = m.a + C * kSP * 4;
  m.total = m.gates + kGateBytes;
  return m;
}

// Eight bf16 values times a bf16 factor: one rounding of the exact product, as in float32 followed by a cast.
__device__ __forceinline__ uint4 scaled_piece(uint4 raw, __nv_bfloat16 factor) {
  const __nv_bfloat162 f2 = __halves2bfloat162(factor, factor);
  auto mul = [&](uint32_t x) {
    const __nv_bfloat162 y = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&x), f2);
    return *reinterpret_cast<const uint32_t*>(&y);
  };
  return make_uint4(mul(raw.x), mul(raw.y), mul(raw.z), mul(raw.w));
}
__device__ __forceinline__ void st_shared16(uint32_t addr, uint4 v) {
  asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

// One CTA per chunk and head, two CTAs per SM.  About 1,300 MMAs per chunk (triangular blocks are skipped) and some 100 KB
// in and out.  Latency-bound (ncu: 0.38 of the issue slots, tensor pipe 0.21).  B=8, S=4096, H=8, K=V=128: 0.225 ms (0.79 ms
// with the products in float32 on the CUDA cores).
template <int KB>
__global__ void __launch_bounds__(kChunkThreads, 2)
fwd_chunk_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k, const __nv_bfloat16* __restrict__ v,
                 const float* __restrict__ g, const __nv_bfloat16* __restrict__ beta, uint8_t* __restrict__ ws, Dims D) {
  extern __shared__ __align__(1024) uint8_t gdn_smem_raw[];
  constexpr ChunkSmem M = chunk_smem(KB);
  const uint32_t base = ptx::smem_u32(gdn_smem_raw);
  if ((base & 1023u) != 0) {
    if (threadIdx.x == 0) raise_status(LEWI_STATUS_SMEM_LAYOUT);
    return;
  }
  const uint32_t tK = base + M.k, tQ = base + M.q, tKb = base + M.kb, tV = base + M.v, tPa = base + M.pa, tPae = base + M.pae;
  float* sS = reinterpret_cast<float*>(gdn_smem_raw + M.s);
  float* sA = reinterpret_cast<float*>(gdn_smem_raw + M.a);
  float* sX = reinterpret_cast<float*>(gdn_smem_raw + M.x);
  float* gates = reinterpret_cast<float*>(gdn_smem_raw + M.gates);
  const int n = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const LaneOff L = lane_off(lane);
  const int K = D.K, V = D.V;
  const long long chunk = ((long long)b * D.N + n) * D.H + h;
  const long long tok0 = (long long)n * C;
  const FwdWs W = fwd_ws(D);
  const __nv_bfloat16 scale = __float2bfloat16_rn(rsqrtf((float)K));
  auto row_off = [&](int r) { return ((long long)b * D.S + tok0 + r) * D.H + h; };   // of token r in units of head rows

  // ---- loads: k, k*beta, q*scale (also to the workspace), the first 128 columns of v*beta; rows past the end are zero.
  // Everything is requested before anything is used: one trip to memory instead of one per array.
  __nv_bfloat16* qs_out = reinterpret_cast<__nv_bfloat16*>(ws + W.qs) + chunk * C * K;
  constexpr int KP8 = KB * 8;   // 16-byte pieces per tile row
  constexpr int NK = C * KP8 / kChunkThreads, NV = C * 16 / kChunkThreads;
  uint4 kr[NK], qr[NK], vr[NV];
  __nv_bfloat16 bk[NK], bv[NV];
  float g0 = 0.f, g1 = 0.f;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  auto fetch_v = [&](int v0) {
#pragma unroll
    for (int x = 0; x < NV; ++x) {
      const int i = x * kChunkThreads + tid, r = i >> 4, p = i & 15;
      const bool in = tok0 + r < D.S && v0 + p * 8 < V;
      vr[x] = in ? ld_nc_v4(v + row_off(r) * V + v0 + p * 8) : zero;
      bv[x] = in ? beta[row_off(r)] : __float2bfloat16_rn(0.f);
    }
  };
  auto place_v = [&]() {
#pragma unroll
    for (int x = 0; x < NV; ++x) {
      const int i = x * kChunkThreads + tid, r = i >> 4, p = i & 15;
      st_shared16(swz(tV + (p >> 3) * kBox, r, p & 7), scaled_piece(vr[x], bv[x]));
    }
  };
  if (warp == 0) {
    if (tok0 + 2 * lane < D.S) g0 = g[row_off(2 * lane)];
    if (tok0 + 2 * lane + 1 < D.S) g1 = g[row_off(2 * lane + 1)];
  }
#pragma unroll
  for (int x = 0; x < NK; ++x) {
    const int i = x * kChunkThreads + tid, r = i / KP8, p = i % KP8;
    const bool in = tok0 + r < D.S && p * 8 < K;
    const long long off = row_off(r) * K + p * 8;
    kr[x] = in ? ld_nc_v4(k + off) : zero;
    qr[x] = in ? ld_nc_v4(q + off) : zero;
    bk[x] = in ? beta[row_off(r)] : __float2bfloat16_rn(0.f);
  }
  fetch_v(0);
  if (warp == 0) chunk_gates(gates, g0, g1, lane);
#pragma unroll
  for (int x = 0; x < NK; ++x) {
    const int i = x * kChunkThreads + tid, r = i / KP8, p = i % KP8;
    const uint4 qsc = scaled_piece(qr[x], scale);
    const uint32_t at = swz((p >> 3) * kBox, r, p & 7);
    st_shared16(tK + at, kr[x]);
    st_shared16(tQ + at, qsc);
    st_shared16(tKb + at, scaled_piece(kr[x], bk[x]));
    if (p * 8 < K) st_v4(qs_out + r * K + p * 8, qsc);
  }
  place_v();
  __syncthreads();
  {
    float* gates_out = reinterpret_cast<float*>(ws + W.gates) + chunk * 3 * C;
    if (tid < 3 * C) gates_out[tid] = gates[tid];
  }

  // ---- S (warps 4-7) and the in-chunk attention (warps 0-3): 16 rows per warp, column tiles up to the diagonal
  {
    const int wm = warp & 3;
    const bool is_s = warp >= 4;
    float acc[8][4];
#pragma unroll
    for (int t = 0; t < 8; ++t) zero4(acc[t]);
#pragma unroll
    for (int ks = 0; ks < 4 * KB; ++ks) {
      const Frag4 a = ld_a(is_s ? tKb : tQ, wm * 16, ks, L);
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        if (p > wm) break;
        mma2_add(acc[2 * p], acc[2 * p + 1], a.r, ld_b(tK, p * 16, ks, L));
      }
    }
    uint32_t* at_out = reinterpret_cast<uint32_t*>(ws + W.attn) + chunk * 3 * C * C / 2;
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      if (t > 2 * wm + 1) break;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int r = wm * 16 + (lane >> 2) + half * 8, c = t * 8 + (lane & 3) * 2;
        const float gr = gates[r];
        float x[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const bool in = is_s ? c + e < r : c + e <= r;
          x[e] = in ? round_bf16(acc[t][half * 2 + e]) * __expf(gr - gates[c + e]) : 0.f;
        }
        if (is_s) {
          *reinterpret_cast<float2*>(sS + r * kSP + c) = make_float2(x[0], x[1]);
        } else {
          uint32_t p0, p1, p2;
          split3(x[0], x[1], p0, p1, p2);
          at_out[(r * C + c) / 2] = p0;
          at_out[(C * C + r * C + c) / 2] = p1;
          at_out[(2 * C * C + r * C + c) / 2] = p2;
        }
      }
    }
  }
  __syncthreads();
  unit_lower_inverse(sS, sA, sX, tid);

  // ---- the pieces of A and of A exp(gcs) (columns scaled), as swizzled tiles
#pragma unroll
  for (int i0 = 0; i0 < C * 8; i0 += kChunkThreads) {
    const int i = i0 + tid, r = i >> 3, p = i & 7;
    const float4 lo = *reinterpret_cast<const float4*>(sA + r * kSP + p * 8), hi = *reinterpret_cast<const float4*>(sA + r * kSP + p * 8 + 4);
    const float a[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    uint32_t pc[3][4];
#pragma unroll
    for (int x = 0; x < 4; ++x) split3(a[2 * x], a[2 * x + 1], pc[0][x], pc[1][x], pc[2][x]);
#pragma unroll
    for (int w3 = 0; w3 < 3; ++w3) st_shared16(swz(tPa + w3 * kBox, r, p), make_uint4(pc[w3][0], pc[w3][1], pc[w3][2], pc[w3][3]));
    const float* e = gates + C + p * 8;
#pragma unroll
    for (int x = 0; x < 4; ++x) split3(a[2 * x] * e[2 * x], a[2 * x + 1] * e[2 * x + 1], pc[0][x], pc[1][x], pc[2][x]);
#pragma unroll
    for (int w3 = 0; w3 < 3; ++w3) st_shared16(swz(tPae + w3 * kBox, r, p), make_uint4(pc[w3][0], pc[w3][1], pc[w3][2], pc[w3][3]));
  }
  __syncthreads();

  // ---- w = (A exp(gcs)) k_beta: every warp takes 8*KB columns of all rows
  {
    __nv_bfloat16* w_out = reinterpret_cast<__nv_bfloat16*>(ws + W.w) + chunk * C * K;
    float acc[4][KB][4];
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int t = 0; t < KB; ++t) zero4(acc[m][t]);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      // the 16-column load covers this warp's columns (KB = 2) or its and its neighbour's (KB = 1)
      const Frag4 bb = ld_b_t(tKb, ks * 16, KB == 2 ? warp : warp >> 1, L);
      float t[4][KB][4];   // (products as Prod2 makes them; four chains side by side)
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int x = 0; x < KB; ++x) zero4(t[m][x]);
#pragma unroll
      for (int w3 = 2; w3 >= 0; --w3)
#pragma unroll
        for (int m = 0; m < 4; ++m) {
          if (m < ks) continue;
          const Frag4 a = ld_a(tPae + w3 * kBox, m * 16, ks, L);
          if constexpr (KB == 2) {
            mma2(t[m][0], t[m][1], a.r, bb);
          } else {
            mma(t[m][0], a.r, (warp & 1) ? bb.r[2] : bb.r[0], (warp & 1) ? bb.r[3] : bb.r[1]);
          }
        }
#pragma unroll
      for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int x = 0; x < KB; ++x) add4(acc[m][x], t[m][x]);
    }
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int t = 0; t < KB; ++t) {
        const int c = warp * 8 * KB + t * 8 + (lane & 3) * 2, r = m * 16 + (lane >> 2);
        if (c < K) {
          *reinterpret_cast<uint32_t*>(w_out + r * K + c) = pack_bf16(acc[m][t][0], acc[m][t][1]);
          *reinterpret_cast<uint32_t*>(w_out + (r + 8) * K + c) = pack_bf16(acc[m][t][2], acc[m][t][3]);
        }
      }
  }
  // ---- u^T = v_beta^T A^T: every warp takes 16 columns of V and all tokens
  for (int v0 = 0; v0 < V; v0 += 128) {
    if (v0 > 0) {
      fetch_v(v0);
      __syncthreads();
      place_v();
      __syncthreads();
    }
    const int blk = v0 / 16 + warp;
    if (blk >= W.v16) continue;
    float acc[8][4];
#pragma unroll
    for (int t = 0; t < 8; ++t) zero4(acc[t]);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const Frag4 a = ld_a_t(tV, ks * 16, warp, L);
      Prod2 x[4];
#pragma unroll
      for (int w3 = 2; w3 >= 0; --w3)
#pragma unroll
        for (int p = 0; p < 4; ++p) {
          if (p < ks) continue;
          x[p].mul(a.r, ld_b(tPa + w3 * kBox, p * 16, ks, L));
        }
#pragma unroll
      for (int p = 0; p < 4; ++p) x[p].add_to(acc[2 * p], acc[2 * p + 1]);
    }
    uint4* out = reinterpret_cast<uint4*>(ws + W.ut) + ((chunk * W.v16 + blk) * 32 + lane) * 4;
#pragma unroll
    for (int x = 0; x < 4; ++x)
      out[x] = make_uint4(pack_bf16(acc[2 * x][0], acc[2 * x][1]), pack_bf16(acc[2 * x][2], acc[2 * x][3]),
                          pack_bf16(acc[2 * x + 1][0], acc[2 * x + 1][1]), pack_bf16(acc[2 * x + 1][2], acc[2 * x + 1][3]));
  }
}

// ------------------------------------------------------------------------------------------------ scan kernel

// One stage of the scan's ring: w, q*scale, k (KB boxes each), the three pieces of the in-chunk attention, the gates.
template <int KB>
struct ScanStage {
  static constexpr int w = 0, q = KB * kBox, k = 2 * KB * kBox, at = 3 * KB * kBox, gates = at + 3 * kBox;
  static constexpr int bytes = gates + 1024;
};
constexpr int kScanStages = 2;
constexpr int kTile = 512;                          // bytes of an accumulator tile: 32 lanes x 4 floats
constexpr int kOutPitch = 48;                       // bytes per token row of a warp's output tile (16 columns; conflict-free)

// Shared memory of the scan: the ring; per column group (16 columns of V, KS warps) the exchange areas for partial v_new
// (KS x 8 tiles) and partial q h (for every warp the other KS - 1 warps' pieces of its 8/KS tiles); output tiles; barriers.
template <int KB, int NG, int KS>
struct ScanSmem {
  static constexpr int own = 8 / KS;                // accumulator tiles (8 tokens each) a warp finishes
  static constexpr int xv = KS > 1 ? KS * 8 * kTile : 0, xo = KS * (KS - 1) * own * kTile, out = C * kOutPitch;
  static constexpr int group = xv + xo + out;
  static constexpr int groups = kScanStages * ScanStage<KB>::bytes;
  static constexpr int bars = groups + NG * group;
  static constexpr int total = bars + 16 * kScanStages + 24 * NG + 16;
};

// Consumer warps plus one producer warp, or - with eight consumers - a producer warpgroup that hands its registers over: a
// ninth warp alone would cap all of them at 168 registers.
constexpr int scan_threads(int warps) { return warps * 32 + (warps == 8 ? 128 : 32); }
// 12 warps x 32 x 168 registers at launch = 64,512 = 8 x 32 x 224 + 4 x 32 x 56
__device__ __forceinline__ void regs_inc224() { asm volatile("setmaxnreg.inc.sync.aligned.u32 224;"); }
__device__ __forceinline__ void regs_dec56() { asm volatile("setmaxnreg.dec.sync.aligned.u32 56;"); }

struct ScanArgs {
  const uint32_t* ut;      // u^T tiles
  const float* gates;
  const float* h0;         // [B,H,K,V] or null
  __nv_bfloat16* o;        // [B,S,H,V]
  float* h_final;          // [B,H,K,V] or null
  float4* hs;              // STATES: state at the start of every chunk, accumulator tiles of h^T [chunks][v16][8*KB][32 lanes]
  float4* vn;              // STATES: v_new, accumulator tiles of v_new^T [chunks][v16][8][32 lanes]
  int v16;
  Dims D;
};

// NG column groups of KS warps.  A group carries 16 columns of the state through the whole sequence, each of its warps K/KS of
// the state's rows, in registers (accumulator layout of h^T).  Per chunk, with operands straight from the accumulators of the
// product before:
//   v^T = u^T - h^T w^T;   o^T = (h^T q^T) exp(gcs) + v^T attn^T;   h^T <- h^T exp(gcs_last) + (v exp(gcs_last - gcs))^T k.
// With KS > 1 the first two products are sums over the group: its warps leave their parts of h^T w^T in shared memory, run the
// q products while the others arrive, and add all parts in the same order; each finishes 64/KS tokens of o.
// 696 m16n8k16 per group and chunk (K = 128), 5,600 cycles of one scheduler at the measured 8 cycles each; a single warp per
// scheduler reached 9,500 (splitting and loading do not overlap its own MMAs), so the launch splits K until every scheduler has
// two warps, or K is in quarters.  B=8, S=4096, H=8, K=V=128: 0.31 ms (1.61 ms in float32 on the CUDA cores), tensor pipe 66 %
// active; B=1, S=1000: 0.035 ms (0.23 ms).
// STATES (the first pass of the gradient): no output; the state at the start of every chunk and v_new are stored instead.
// A producer warp keeps a ring of two chunks filled by TMA: issuing the nine copies takes a thousand cycles, which the other
// warps of a group would spend waiting for the one that does it.
template <int KB, int NG, int KS, bool STATES>
__device__ __forceinline__ void fwd_scan(const CUtensorMap& tm_w, const CUtensorMap& tm_q, const CUtensorMap& tm_k, const CUtensorMap& tm_at,
                                         const ScanArgs& a, int cta_x) {
  extern __shared__ __align__(1024) uint8_t gdn_smem_raw[];
  using St = ScanStage<KB>;
  using Sm = ScanSmem<KB, NG, KS>;
  constexpr int KT = 4 * KB / KS;         // this warp's 16-deep steps over K
  constexpr int OWN = Sm::own, OP = OWN / 2;   // tiles and tile pairs of o that this warp finishes
  const uint32_t base = ptx::smem_u32(gdn_smem_raw);
  if ((base & 1023u) != 0) {
    if (threadIdx.x == 0) raise_status(LEWI_STATUS_SMEM_LAYOUT);
    return;
  }
  const uint32_t bars = base + Sm::bars;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (kScanStages + s); };
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gdn_smem_raw + Sm::total - 16);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const LaneOff L = lane_off(lane);
  const int grp = warp / KS, kq = warp % KS;
  const int h = blockIdx.y, b = blockIdx.z;
  const Dims& D = a.D;
  const uint32_t grp_bars = bars + 16 * kScanStages + 24 * grp;   // of this group: parts of v there, parts of o there, area free
  const uint32_t v_bar = grp_bars, o_bar = grp_bars + 8, free_bar = grp_bars + 16;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kScanStages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), NG * KS);
    }
    for (int x = 0; x < 3 * NG; ++x) ptx::mbar_init(bars + 16 * kScanStages + 8 * x, KS);
    *abort_flag = 0;
    ptx::mbar_fence_init();
    ptx::fence_proxy_async();
  }
  __syncthreads();

  constexpr int NW = NG * KS;   // consumer warps
  if (warp >= NW) {
    if constexpr (NW == 8) regs_dec56();
    if (warp == NW && lane == 0) {
      int n = 0;
      for (; n < D.N; ++n) {
        const int s = n % kScanStages;
        if (n >= kScanStages && !ptx::mbar_wait(empty_bar(s), ((n / kScanStages) & 1u) ^ 1u, abort_flag)) break;
        const uint32_t st = base + s * St::bytes, fb = full_bar(s);
        const int chunk = (b * D.N + n) * D.H + h;
        ptx::mbar_expect_tx(fb, (STATES ? 2 * KB : 3 * KB + 3) * kBox + kGateBytes);
#pragma unroll
        for (int x = 0; x < KB; ++x) ptx::tma_load_2d(st + St::w + x * kBox, &tm_w, fb, 64 * x, chunk * C);
        if constexpr (!STATES) {
#pragma unroll
          for (int x = 0; x < KB; ++x) ptx::tma_load_2d(st + St::q + x * kBox, &tm_q, fb, 64 * x, chunk * C);
          ptx::tma_load_2d(st + St::at, &tm_at, fb, 0, chunk * 3 * C);
        }
        ptx::bulk_load(st + St::gates, a.gates + (long long)chunk * 3 * C, fb, kGateBytes);
#pragma unroll
        for (int x = 0; x < KB; ++x) ptx::tma_load_4d(st + St::k + x * kBox, &tm_k, fb, 64 * x, h, n * C, b);
      }
      if (*abort_flag) {   // copies in flight land (bounded) before the CTA goes
        const unsigned long long t0 = ptx::globaltimer_ns();
        for (int j = max(0, n - kScanStages); j < n; ++j)
          while (!ptx::mbar_try_wait(full_bar(j % kScanStages), (j / kScanStages) & 1u) && ptx::globaltimer_ns() - t0 < 4000000ull) {
          }
      }
    }
    __syncthreads();
    return;
  }
  if constexpr (NW == 8) regs_inc224();
  const int blk = cta_x * NG + grp;    // 16 columns of V
  const bool live = blk < a.v16;
  const int vr = blk * 16 + (lane >> 2);    // this lane's columns of V: vr and vr + 8
  const int kc = (lane & 3) * 2;            // its place within every 8 tokens / state rows
  const int k0 = kq * KT * 16;              // first state row of this warp
  const long long hbase = ((long long)b * D.H + h) * D.K * D.V;
  // token pairs (16 tokens) in this warp's order: the OP pairs it finishes first; pairs are dealt so that the triangular
  // attention product is even (KS = 2: 0,3 | 1,2)
  auto pair_at = [&](int i) { return KS == 2 ? (i < 2 ? (kq == 0 ? 3 * i : 1 + i) : (kq == 0 ? i - 1 : 3 * (i - 2))) : ((kq + i) & 3); };
  float hh[2 * KT][4];
#pragma unroll
  for (int t = 0; t < 2 * KT; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int kk = k0 + t * 8 + kc + (e & 1), vv = vr + (e >> 1) * 8;
      hh[t][e] = (a.h0 != nullptr && kk < D.K && vv < D.V) ? a.h0[hbase + (long long)kk * D.V + vv] : 0.f;
    }
  auto u_at = [&](int n) { return reinterpret_cast<const uint4*>(a.ut) + ((((long long)b * D.N + n) * D.H + h) * a.v16 + blk) * 128 + lane * 4; };
  uint4 u_next[4];
#pragma unroll
  for (int x = 0; x < 4; ++x) u_next[x] = live ? u_at(0)[x] : make_uint4(0, 0, 0, 0);
  uint8_t* xv = gdn_smem_raw + Sm::groups + grp * Sm::group;
  uint8_t* xo = xv + Sm::xv;
  uint8_t* my_out = xo + Sm::xo + kq * (C / KS) * kOutPitch;
  bool ok = true;
  for (int n = 0; n < D.N; ++n) {
    const int s = n % kScanStages;
    ok = ptx::mbar_wait(full_bar(s), (n / kScanStages) & 1u, abort_flag);
    if (!__all_sync(0xffffffffu, ok)) break;
    if (!live) {   // a warp past the last column only keeps the ring moving
      if (lane == 0) ptx::mbar_arrive(empty_bar(s));
      continue;
    }
    const uint32_t st = base + s * St::bytes;
    const float* gates = reinterpret_cast<const float*>(gdn_smem_raw + s * St::bytes + St::gates);
    uint4 u_cur[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) u_cur[x] = u_next[x];
    if (n + 1 < D.N) {
#pragma unroll
      for (int x = 0; x < 4; ++x) u_next[x] = u_at(n + 1)[x];
    }
    if constexpr (STATES) {
      float4* dst = a.hs + (((((long long)b * D.N + n) * D.H + h) * a.v16 + blk) * (8 * KB) + kq * 2 * KT) * 32 + lane;
#pragma unroll
      for (int t = 0; t < 2 * KT; ++t) dst[t * 32] = make_float4(hh[t][0], hh[t][1], hh[t][2], hh[t][3]);
    }
    // h^T w^T with the old state (summed up by the tensor core, here and in rev_scan: with rounded sums the state is as far from 64 bits)
    float vn[8][4];
#pragma unroll
    for (int t = 0; t < 8; ++t) zero4(vn[t]);
    Frag3x4 hf[KT];
#pragma unroll
    for (int ks = 0; ks < KT; ++ks) {
      split_acc(hh[2 * ks], hh[2 * ks + 1], hf[ks]);
#pragma unroll
      for (int p = 0; p < 4; p += 2) {
        const Frag4 b0 = ld_b(st + St::w, p * 16, kq * KT + ks, L), b1 = ld_b(st + St::w, p * 16 + 16, kq * KT + ks, L);
#pragma unroll
        for (int w3 = 2; w3 >= 0; --w3) {
          mma2(vn[2 * p], vn[2 * p + 1], hf[ks].p[w3], b0);
          mma2(vn[2 * p + 2], vn[2 * p + 3], hf[ks].p[w3], b1);
        }
      }
    }
    if constexpr (KS > 1) {
      if (n > 0) ok = ptx::mbar_wait(free_bar, (n - 1) & 1u, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) break;
#pragma unroll
      for (int t = 0; t < 8; ++t)
        *reinterpret_cast<float4*>(xv + (kq * 8 + t) * kTile + lane * 16) = make_float4(vn[t][0], vn[t][1], vn[t][2], vn[t][3]);
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(v_bar);
    }
    // h^T q^T
    float oo[8][4];
    if constexpr (!STATES) {
#pragma unroll
      for (int t = 0; t < 8; ++t) zero4(oo[t]);
#pragma unroll
      for (int ks = 0; ks < KT; ++ks)
#pragma unroll
        for (int i = 0; i < 4; i += 2) {
          const Frag4 b0 = ld_b(st + St::q, pair_at(i) * 16, kq * KT + ks, L), b1 = ld_b(st + St::q, pair_at(i + 1) * 16, kq * KT + ks, L);
#pragma unroll
          for (int w3 = 2; w3 >= 0; --w3) {   // (o is rounded to bf16: accumulated by the tensor core)
            mma2(oo[2 * i], oo[2 * i + 1], hf[ks].p[w3], b0);
            mma2(oo[2 * i + 2], oo[2 * i + 3], hf[ks].p[w3], b1);
          }
        }
      if constexpr (KS > 1) {
        // tiles that another warp finishes go to that warp's slots; slot order: the sender's distance
#pragma unroll
        for (int t = OWN; t < 8; ++t) {
          const int d = t / OWN, to = KS == 2 ? kq ^ 1 : (kq + d) & (KS - 1);
          *reinterpret_cast<float4*>(xo + ((to * (KS - 1) + d - 1) * OWN + t % OWN) * kTile + lane * 16) =
              make_float4(oo[t][0], oo[t][1], oo[t][2], oo[t][3]);
        }
        __syncwarp();
        if (lane == 0) ptx::mbar_arrive(o_bar);
      }
    }
    // v_new = u - w h: all parts in the same order in every warp
    if constexpr (KS > 1) {
      ok = ptx::mbar_wait(v_bar, n & 1u, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) break;
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const float4 x = *reinterpret_cast<const float4*>(xv + ((kq ^ 1) * 8 + t) * kTile + lane * 16);
        vn[t][0] += x.x; vn[t][1] += x.y; vn[t][2] += x.z; vn[t][3] += x.w;
        if constexpr (KS == 4) {
          const float4 y = *reinterpret_cast<const float4*>(xv + ((kq ^ 2) * 8 + t) * kTile + lane * 16);
          const float4 z = *reinterpret_cast<const float4*>(xv + ((kq ^ 3) * 8 + t) * kTile + lane * 16);
          vn[t][0] += y.x + z.x; vn[t][1] += y.y + z.y; vn[t][2] += y.z + z.z; vn[t][3] += y.w + z.w;
        }
      }
    }
    const uint32_t* uu = reinterpret_cast<const uint32_t*>(u_cur);
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      vn[t][0] = bf16_lo(uu[2 * t]) - vn[t][0];
      vn[t][1] = bf16_hi(uu[2 * t]) - vn[t][1];
      vn[t][2] = bf16_lo(uu[2 * t + 1]) - vn[t][2];
      vn[t][3] = bf16_hi(uu[2 * t + 1]) - vn[t][3];
    }
    if constexpr (STATES) {
      float4* dst = a.vn + ((((long long)b * D.N + n) * D.H + h) * a.v16 + blk) * 8 * 32 + lane;
#pragma unroll
      for (int t = 0; t < 8; ++t)
        if (KS == 1 || t / OWN == kq) dst[t * 32] = make_float4(vn[t][0], vn[t][1], vn[t][2], vn[t][3]);
    }
    const float dec = gates[2 * C - 1];
    // attn v_new, 16 tokens of v_new at a time; the pieces of v_new exp(gcs_last - gcs)
    Frag3x4 sf[4];
    float oa[OWN][4];
#pragma unroll
    for (int t = 0; t < OWN; ++t) zero4(oa[t]);
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      Frag3x4 vf;
      if constexpr (!STATES) split_acc(vn[2 * ks], vn[2 * ks + 1], vf);
#pragma unroll
      for (int i = 0; i < (STATES ? 0 : OP); ++i) {
        const int p = pair_at(i);
        if (p < ks) continue;   // attn is lower triangular: tokens 16*ks.. reach rows from 16*ks on
        const Frag4 b[3] = {ld_b(st + St::at, p * 16, ks, L), ld_b(st + St::at + kBox, p * 16, ks, L), ld_b(st + St::at + 2 * kBox, p * 16, ks, L)};
        mma2_x6_acc(oa[2 * i], oa[2 * i + 1], vf, b);
      }
#pragma unroll
      for (int t = 2 * ks; t < 2 * ks + 2; ++t) {
        const float2 e = *reinterpret_cast<const float2*>(gates + 2 * C + t * 8 + kc);
        vn[t][0] *= e.x; vn[t][1] *= e.y; vn[t][2] *= e.x; vn[t][3] *= e.y;
      }
      split_acc(vn[2 * ks], vn[2 * ks + 1], sf[ks]);
    }
    // h = h exp(gcs_last) + (k exp(gcs_last - gcs))^T v_new
    constexpr int CW = KT >= 2 ? 2 : 1;   // column pairs side by side: independent accumulators between dependent MMAs
#pragma unroll
    for (int cp = 0; cp < KT; cp += CW) {
      float add[2 * CW][4];
      chunk_sum<CW>(add, sf, [&](int ks, int x) { return ld_b_t(st + St::k, ks * 16, kq * KT + cp + x, L); });
#pragma unroll
      for (int t = 0; t < 2 * CW; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) hh[2 * cp + t][e] = fmaf(hh[2 * cp + t][e], dec, add[t][e]);
    }
    if constexpr (STATES) {   // (a quicker warp may not overwrite parts of v_new that a slower one still reads)
      __syncwarp();
      if (lane == 0) {
        if (KS > 1) ptx::mbar_arrive(free_bar);
        ptx::mbar_arrive(empty_bar(s));
      }
      continue;
    }
    // o = (q h) exp(gcs) + attn v_new
    if constexpr (KS > 1) {
      ok = ptx::mbar_wait(o_bar, n & 1u, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) break;
#pragma unroll
      for (int t = 0; t < OWN; ++t)
#pragma unroll
        for (int d = KS - 2; d >= 0; --d) {
          const float4 x = *reinterpret_cast<const float4*>(xo + ((kq * (KS - 1) + d) * OWN + t) * kTile + lane * 16);
          oo[t][0] += x.x; oo[t][1] += x.y; oo[t][2] += x.z; oo[t][3] += x.w;
        }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(free_bar);
    }
#pragma unroll
    for (int t = 0; t < OWN; ++t) {
      const float2 e = *reinterpret_cast<const float2*>(gates + C + (2 * pair_at(t >> 1) + (t & 1)) * 8 + kc);
      oo[t][0] = fmaf(oo[t][0], e.x, oa[t][0]); oo[t][1] = fmaf(oo[t][1], e.y, oa[t][1]);
      oo[t][2] = fmaf(oo[t][2], e.x, oa[t][2]); oo[t][3] = fmaf(oo[t][3], e.y, oa[t][3]);
    }
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(empty_bar(s));
    // transposed through this warp's tile, 16-byte stores (two lanes per token)
#pragma unroll
    for (int i = 0; i < OP; ++i)
      stsm_t(ptx::smem_u32(my_out) + (16 * i + ((lane >> 4) << 3) + (lane & 7)) * kOutPitch + ((lane >> 3) & 1) * 16,
             pack_bf16(oo[2 * i][0], oo[2 * i][1]), pack_bf16(oo[2 * i][2], oo[2 * i][3]),
             pack_bf16(oo[2 * i + 1][0], oo[2 * i + 1][1]), pack_bf16(oo[2 * i + 1][2], oo[2 * i + 1][3]));
    __syncwarp();
    const int vcol = blk * 16 + (lane & 1) * 8;
#pragma unroll
    for (int i = 0; i < OP; ++i) {
      const long long t = (long long)n * C + pair_at(i) * 16 + (lane >> 1);
      const uint4 val = *reinterpret_cast<const uint4*>(my_out + (i * 16 + (lane >> 1)) * kOutPitch + (lane & 1) * 16);
      if (t < D.S && vcol < D.V) st_out8(a.o + (((long long)b * D.S + t) * D.H + h) * D.V + vcol, val, a.o);
    }
    __syncwarp();
  }
  if (a.h_final != nullptr && live && ok) {
#pragma unroll
    for (int t = 0; t < 2 * KT; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int kk = k0 + t * 8 + kc + (e & 1), vv = vr + (e >> 1) * 8;
        if (kk < D.K && vv < D.V) a.h_final[hbase + (long long)kk * D.V + vv] = hh[t][e];
      }
  }
  __syncthreads();
}

template <int KB, int NG, int KS>
__global__ void __launch_bounds__(scan_threads(NG * KS), 1)
fwd_scan_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                const __grid_constant__ CUtensorMap tm_at, const ScanArgs a) {
  fwd_scan<KB, NG, KS, false>(tm_w, tm_q, tm_k, tm_at, a, blockIdx.x);
}

// ------------------------------------------------------------------------------------------------ host side

// [rows][64-column boxes] view of a bf16 matrix with `cols` columns: boxes of `box_rows` x 64, columns past the end are zero
inline bool rows_map(CUtensorMap* m, const void* ptr, int cols, long long rows, int box_rows) {
  return gg::make_map(m, ptr, (uint64_t)cols, (uint64_t)rows, 0, 64, (uint32_t)box_rows);
}
// a [B,S,H,W] bf16 tensor: boxes of 64 tokens x 64 columns of one head; tokens and columns past the end are zero
inline bool heads_map(CUtensorMap* m, const void* ptr, int B, int S, int H, int W) {
  const cuuint64_t dims[4] = {(cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)S, (cuuint64_t)B};
  const cuuint64_t strides[3] = {(cuuint64_t)W * 2, (cuuint64_t)W * H * 2, (cuuint64_t)W * H * S * 2};
  const cuuint32_t box[4] = {64, 1, 64, 1};
  return gg::encode_tiled(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, ptr, dims, strides, box);
}

template <int KB>
inline int launch_chunk(cudaStream_t st, const void* q, const void* k, const void* v, const float* g, const void* beta, uint8_t* ws,
                        const Dims& D) {
  static bool done[64] = {false};
  constexpr int smem = chunk_smem(KB).total;
  if (!allow_smem(fwd_chunk_kernel<KB>, smem, done)) return LEWI_ERR_CUDA;
  fwd_chunk_kernel<KB><<<dim3((unsigned)D.N, (unsigned)D.H, (unsigned)D.B), kChunkThreads, smem, st>>>(
      reinterpret_cast<const __nv_bfloat16*>(q), reinterpret_cast<const __nv_bfloat16*>(k), reinterpret_cast<const __nv_bfloat16*>(v), g,
      reinterpret_cast<const __nv_bfloat16*>(beta), ws, D);
  LEWI_CHECK_LAUNCH();
  return LEWI_OK;
}

struct ScanMaps {
  CUtensorMap w, q, k, at;
};

template <int KB, int NG, int KS>
inline int launch_scan(cudaStream_t st, const ScanMaps& m, const ScanArgs& a) {
  static bool done[64] = {false};
  constexpr int smem = ScanSmem<KB, NG, KS>::total;
  if (!allow_smem(fwd_scan_kernel<KB, NG, KS>, smem, done)) return LEWI_ERR_CUDA;
  fwd_scan_kernel<KB, NG, KS><<<dim3((unsigned)((a.v16 + NG - 1) / NG), (unsigned)a.D.H, (unsigned)a.D.B), scan_threads(NG * KS), smem, st>>>(
      m.w, m.q, m.k, m.at, a);
  LEWI_CHECK_LAUNCH();
  return LEWI_OK;
}

// Column groups per scan CTA: the fewest that still give every CTA an SM of its own (a CTA's groups share the loads).
inline int scan_groups(const Dims& D, int v16) {
  for (int ng = 1; ng < 8; ng *= 2)
    if ((long long)D.B * D.H * ((v16 + ng - 1) / ng) <= num_sms()) return ng;
  return 8;
}

// `a` says what is read and written; the tensor maps come from the forward workspace.
template <int KB>
inline int scan(cudaStream_t st, const void* k, const uint8_t* ws, const ScanArgs& a) {
  const Dims& D = a.D;
  const FwdWs W = fwd_ws(D);
  const long long rows = (long long)D.B * D.N * D.H * C;
  ScanMaps m;
  if (!rows_map(&m.w, ws + W.w, D.K, rows, C) || !rows_map(&m.q, ws + W.qs, D.K, rows, C) || !heads_map(&m.k, k, D.B, D.S, D.H, D.K) ||
      !rows_map(&m.at, ws + W.attn, C, 3 * rows, 3 * C))
    return LEWI_ERR_CUDA;
  switch (scan_groups(D, W.v16)) {   // 4, 8, 8 and 8 warps: two per scheduler once there are enough columns
    case 1: return launch_scan<KB, 1, 4>(st, m, a);
    case 2: return launch_scan<KB, 2, 4>(st, m, a);
    case 4: return launch_scan<KB, 4, 2>(st, m, a);
    default: return launch_scan<KB, 8, 1>(st, m, a);
  }
}

template <int KB>
inline int forward(cudaStream_t st, const void* q, const void* k, const void* v, const float* g, const void* beta, const float* h0, void* o,
                   float* h_final, uint8_t* ws, const Dims& D) {
  if (int rc = launch_chunk<KB>(st, q, k, v, g, beta, ws, D)) return rc;
  const FwdWs W = fwd_ws(D);
  const ScanArgs a{reinterpret_cast<const uint32_t*>(ws + W.ut), reinterpret_cast<const float*>(ws + W.gates), h0,
                   reinterpret_cast<__nv_bfloat16*>(o), h_final, nullptr, nullptr, W.v16, D};
  return scan<KB>(st, k, ws, a);
}

}  // namespace gdn
}  // namespace lewi
