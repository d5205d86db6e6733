// Chunked gated delta rule, backward.  Forward definitions and notation: gdn_fwd.cuh.
//
// The roundings to bf16 of the forward pass are kept in the values and treated as the identity in the derivative
// (what automatic differentiation of the reference's forward does with its casts).  Per chunk, with
//   kb = bf16(k beta), vb = bf16(v beta), E = exp(gcs), D_ij = exp(gcs_i - gcs_j), kg = kb E, qE = q E,
//   kd = k exp(gcs_last - gcs), S = strict(bf16(kb k^T) D), A = (I + S)^-1, u = bf16(A vb), w = bf16(A kg),
//   P = bf16(q k^T), attn = lower(P D), v_new = u - w h_in,
// and the upstream gradients do (of o) and dh (of the state after the chunk):
//   dv_new = attn^T do + kd dh                      dh_in = qE^T do + dh exp(gcs_last) - w^T dv_new
//   dattn  = lower(do v_new^T), T = dattn D         dqE = do h_in^T      dkd = v_new dh^T
//   dvb = A^T dv_new                                dkg = A^T dw = -dvb h_in^T                (dw = -dv_new h_in^T)
//   dq = (dqE E + T k) scale                        dk = dkd exp(gcs_last - gcs) + T^T q + dP^T kb + dkb beta
//   dS = -strict(X A^T), X = A^T dA = dvb vb^T + dkg kg^T        dP = dS D        dkb = dkg E + dP k
//   dv = dvb beta               dbeta = rowsum(dkb k) + rowsum(dvb v)
//   dgcs = rowsum(dqE qE) - rowsum(dkd kd) + rowsum(G) - colsum(G) + rowsum(dkg kg)      with G = T P + dS S,
//   dgcs_last += exp(gcs_last) <dh, h_in> + sum(dkd kd);        dg = reverse cumulative sum of dgcs inside the chunk.
//
// Two kernels, no atomics: the forward scan again, storing h_in and v_new of every chunk (gdn_fwd.cuh), beside the same scan in
// reverse for dv_new and dh; then one CTA per chunk and head for everything else.  (A^T dA through dvb and dkg, and dkg
// through dvb, save the products dw, dv_new vb^T, dw kg^T and A^T dw of the direct order, half of that kernel's work.)
#pragma once

#include "gdn_fwd.cuh"

namespace lewi {
namespace gdn {

constexpr int kMaxVBwd = 128;

// Backward workspace: accumulator tiles (32 lanes x 4 floats) of the transposed matrices, as the scans hold them:
//   hs, dh [chunks][v16][8*kboxes][32] tiles of h_in^T and of dh^T (16 columns of V by 8 rows of the state each)
//   vn, dv [chunks][v16][8][32]        tiles of v_new^T and dv_new^T (16 columns of V by 8 tokens)
// and room for a copy of do, which the reverse scan fetches by TMA: made where do does not lie on a 16-byte boundary.
struct BwdWs {
  long long hs, dh, vn, dv, d_o, total;
  int v16, kboxes;
};
__host__ __device__ inline BwdWs bwd_ws(const Dims& D) {
  BwdWs o;
  const long long chunks = (long long)D.B * D.N * D.H;
  o.v16 = (D.V + 15) / 16;
  o.kboxes = (D.K + 63) / 64;
  const long long state = chunks * o.v16 * 8 * o.kboxes * 512, rows = chunks * o.v16 * 8 * 512;
  o.hs = 0;
  o.dh = state;
  o.vn = 2 * state;
  o.dv = 2 * state + rows;
  o.d_o = 2 * (state + rows);
  o.total = o.d_o + ((long long)D.B * D.S * D.H * D.V * 2 + 255) / 256 * 256;
  return o;
}

// ------------------------------------------------------------------------------------------------ reverse scan

template <int KB, int NG>
struct RevStage {
  static constexpr int dboxes = NG == 8 ? 2 : 1;    // 64-column boxes of do that the CTA's columns lie in
  static constexpr int w = 0, q = KB * kBox, k = 2 * KB * kBox, at = 3 * KB * kBox, d_o = at + 3 * kBox, gates = d_o + dboxes * kBox;
  static constexpr int bytes = gates + 1024;
};
template <int KB, int NG, int KS>
struct RevSmem {
  static constexpr int xv = KS > 1 ? KS * 8 * kTile : 0;
  static constexpr int groups = kScanStages * RevStage<KB, NG>::bytes;
  static constexpr int bars = groups + NG * xv;
  static constexpr int total = bars + 16 * kScanStages + 16 * NG + 16;
};

struct RevArgs {
  const float* gates;
  const float* dh_final;   // [B,H,K,V] or null
  float* dh0;              // [B,H,K,V] or null
  float4* dh;              // dh at the end of every chunk
  float4* dv;              // dv_new
  int v16;
  Dims D;
};

// The forward scan's structure with dh^T in the registers and the chunks in reverse:
//   dv^T = (dh^T k^T) exp(gcs_last - gcs) + do^T attn;   dh^T <- dh^T exp(gcs_last) + (do exp(gcs))^T q - dv^T w.
// Token pairs (16 tokens) are kept in the warp's own order throughout, the OP pairs that it finishes first.
// 636 m16n8k16 per group and chunk at K = 128.  B=8, S=4096, H=8, K=V=128: 0.31 ms, the forward pass before it 0.20 ms (both
// together 6.7 ms in float32 on the CUDA cores).
template <int KB, int NG, int KS>
__device__ __forceinline__ void rev_scan(const CUtensorMap& tm_w, const CUtensorMap& tm_q, const CUtensorMap& tm_k, const CUtensorMap& tm_at,
                                         const CUtensorMap& tm_do, const RevArgs& a, int cta_x) {
  extern __shared__ __align__(1024) uint8_t gdn_smem_raw[];
  using St = RevStage<KB, NG>;
  using Sm = RevSmem<KB, NG, KS>;
  constexpr int KT = 4 * KB / KS, OWN = 8 / KS, OP = OWN / 2, NW = NG * KS;
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
  const uint32_t v_bar = bars + 16 * kScanStages + 16 * grp, free_bar = v_bar + 8;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kScanStages; ++s) {
      ptx::mbar_init(full_bar(s), 1);
      ptx::mbar_init(empty_bar(s), NW);
    }
    for (int x = 0; x < 2 * NG; ++x) ptx::mbar_init(bars + 16 * kScanStages + 8 * x, KS);
    *abort_flag = 0;
    ptx::mbar_fence_init();
    ptx::fence_proxy_async();
  }
  __syncthreads();
  if (warp >= NW) {
    if constexpr (NW == 8) regs_dec56();
    if (warp == NW && lane == 0) {
      const int d_col = cta_x * NG / 4 * 64;   // first do column of the CTA's boxes
      int it = 0;
      for (; it < D.N; ++it) {
        const int s = it % kScanStages, n = D.N - 1 - it;
        if (it >= kScanStages && !ptx::mbar_wait(empty_bar(s), ((it / kScanStages) & 1u) ^ 1u, abort_flag)) break;
        const uint32_t st = base + s * St::bytes, fb = full_bar(s);
        const int chunk = (b * D.N + n) * D.H + h;
        ptx::mbar_expect_tx(fb, (3 * KB + 3 + St::dboxes) * kBox + kGateBytes);
#pragma unroll
        for (int x = 0; x < KB; ++x) ptx::tma_load_4d(st + St::k + x * kBox, &tm_k, fb, 64 * x, h, n * C, b);
        ptx::bulk_load(st + St::gates, a.gates + (long long)chunk * 3 * C, fb, kGateBytes);
#pragma unroll
        for (int x = 0; x < St::dboxes; ++x) ptx::tma_load_4d(st + St::d_o + x * kBox, &tm_do, fb, d_col + 64 * x, h, n * C, b);
        ptx::tma_load_2d(st + St::at, &tm_at, fb, 0, chunk * 3 * C);
#pragma unroll
        for (int x = 0; x < KB; ++x) ptx::tma_load_2d(st + St::q + x * kBox, &tm_q, fb, 64 * x, chunk * C);
#pragma unroll
        for (int x = 0; x < KB; ++x) ptx::tma_load_2d(st + St::w + x * kBox, &tm_w, fb, 64 * x, chunk * C);
      }
      if (*abort_flag) {   // copies in flight land (bounded) before the CTA goes
        const unsigned long long t0 = ptx::globaltimer_ns();
        for (int j = max(0, it - kScanStages); j < it; ++j)
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
  const int dp = NG == 8 ? grp : (blk & 3); // this group's 16 columns within the do boxes
  const int vr = blk * 16 + (lane >> 2), kc = (lane & 3) * 2, k0 = kq * KT * 16;
  const long long hbase = ((long long)b * D.H + h) * D.K * D.V;
  auto pair_at = [&](int i) { return KS == 2 ? (i < 2 ? (kq == 0 ? 3 * i : 1 + i) : (kq == 0 ? i - 1 : 3 * (i - 2))) : ((kq + i) & 3); };
  float dh[2 * KT][4];
#pragma unroll
  for (int t = 0; t < 2 * KT; ++t)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int kk = k0 + t * 8 + kc + (e & 1), vv = vr + (e >> 1) * 8;
      dh[t][e] = (a.dh_final != nullptr && kk < D.K && vv < D.V) ? a.dh_final[hbase + (long long)kk * D.V + vv] : 0.f;
    }
  uint8_t* xv = gdn_smem_raw + Sm::groups + grp * Sm::xv;
  bool ok = true;
  for (int it = 0; it < D.N; ++it) {
    const int s = it % kScanStages, n = D.N - 1 - it;
    ok = ptx::mbar_wait(full_bar(s), (it / kScanStages) & 1u, abort_flag);
    if (!__all_sync(0xffffffffu, ok)) break;
    if (!live) {
      if (lane == 0) ptx::mbar_arrive(empty_bar(s));
      continue;
    }
    const uint32_t st = base + s * St::bytes;
    const float* gates = reinterpret_cast<const float*>(gdn_smem_raw + s * St::bytes + St::gates);
    const long long tile0 = (((long long)b * D.N + n) * D.H + h) * a.v16 + blk;
    float4* dh_out = a.dh + (tile0 * (8 * KB) + kq * 2 * KT) * 32 + lane;
#pragma unroll
    for (int t = 0; t < 2 * KT; ++t) dh_out[t * 32] = make_float4(dh[t][0], dh[t][1], dh[t][2], dh[t][3]);
    // (dh^T k^T) exp(gcs_last - gcs) over this warp's rows of the state
    float dv[8][4];
#pragma unroll
    for (int t = 0; t < 8; ++t) zero4(dv[t]);
#pragma unroll
    for (int ks = 0; ks < KT; ++ks) {
      Frag3x4 hf;
      split_acc(dh[2 * ks], dh[2 * ks + 1], hf);
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        const Frag4 b0 = ld_b(st + St::k, pair_at(i) * 16, kq * KT + ks, L), b1 = ld_b(st + St::k, pair_at(i + 1) * 16, kq * KT + ks, L);
#pragma unroll
        for (int w3 = 2; w3 >= 0; --w3) {
          mma2(dv[2 * i], dv[2 * i + 1], hf.p[w3], b0);
          mma2(dv[2 * i + 2], dv[2 * i + 3], hf.p[w3], b1);
        }
      }
    }
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      const float2 e = *reinterpret_cast<const float2*>(gates + 2 * C + pair_at(t >> 1) * 16 + (t & 1) * 8 + kc);
      dv[t][0] *= e.x; dv[t][1] *= e.y; dv[t][2] *= e.x; dv[t][3] *= e.y;
    }
    // do^T attn for the tokens this warp finishes: attn is lower triangular, tokens i >= j
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const Frag4 da = ld_a_t(st + St::d_o, ks * 16, dp, L);
#pragma unroll
      for (int i = 0; i < OP; ++i) {
        const int p = pair_at(i);
        if (p > ks) continue;
        const Frag4 b[3] = {ld_b_t(st + St::at, ks * 16, p, L), ld_b_t(st + St::at + kBox, ks * 16, p, L), ld_b_t(st + St::at + 2 * kBox, ks * 16, p, L)};
        mma2_x3(dv[2 * i], dv[2 * i + 1], da.r, b);
      }
    }
    if constexpr (KS > 1) {
      if (it > 0) ok = ptx::mbar_wait(free_bar, (it - 1) & 1u, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) break;
#pragma unroll
      for (int t = 0; t < 8; ++t)
        *reinterpret_cast<float4*>(xv + (kq * 8 + 2 * pair_at(t >> 1) + (t & 1)) * kTile + lane * 16) = make_float4(dv[t][0], dv[t][1], dv[t][2], dv[t][3]);
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(v_bar);
    }
    // dh = dh exp(gcs_last) + (do exp(gcs))^T q, while the other warps' parts of dv arrive
    const float dec = gates[2 * C - 1];
    constexpr int CW = KT >= 2 ? 2 : 1;   // column pairs side by side
    Frag3x4 af[4];
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const Frag4 da = ld_a_t(st + St::d_o, ks * 16, dp, L);
      const float2 e0 = *reinterpret_cast<const float2*>(gates + C + ks * 16 + kc), e1 = *reinterpret_cast<const float2*>(gates + C + ks * 16 + 8 + kc);
#pragma unroll
      for (int x = 0; x < 4; ++x) {
        const float2 e = x < 2 ? e0 : e1;
        split3(bf16_lo(da.r[x]) * e.x, bf16_hi(da.r[x]) * e.y, af[ks].p[0][x], af[ks].p[1][x], af[ks].p[2][x]);
      }
    }
#pragma unroll
    for (int cp = 0; cp < KT; cp += CW) {
      float add[2 * CW][4];
      chunk_sum<CW>(add, af, [&](int ks, int x) { return ld_b_t(st + St::q, ks * 16, kq * KT + cp + x, L); });
#pragma unroll
      for (int t = 0; t < 2 * CW; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) dh[2 * cp + t][e] = fmaf(dh[2 * cp + t][e], dec, add[t][e]);
    }
    if constexpr (KS > 1) {
      ok = ptx::mbar_wait(v_bar, it & 1u, abort_flag);
      if (!__all_sync(0xffffffffu, ok)) break;
#pragma unroll
      for (int t = 0; t < 8; ++t) {
        const int at = 2 * pair_at(t >> 1) + (t & 1);
        const float4 x = *reinterpret_cast<const float4*>(xv + ((kq ^ 1) * 8 + at) * kTile + lane * 16);
        dv[t][0] += x.x; dv[t][1] += x.y; dv[t][2] += x.z; dv[t][3] += x.w;
        if constexpr (KS == 4) {
          const float4 y = *reinterpret_cast<const float4*>(xv + ((kq ^ 2) * 8 + at) * kTile + lane * 16);
          const float4 z = *reinterpret_cast<const float4*>(xv + ((kq ^ 3) * 8 + at) * kTile + lane * 16);
          dv[t][0] += y.x + z.x; dv[t][1] += y.y + z.y; dv[t][2] += y.z + z.z; dv[t][3] += y.w + z.w;
        }
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(free_bar);
    }
    float4* dv_out = a.dv + tile0 * 8 * 32 + lane;
#pragma unroll
    for (int t = 0; t < OWN; ++t) dv_out[(2 * pair_at(t >> 1) + (t & 1)) * 32] = make_float4(dv[t][0], dv[t][1], dv[t][2], dv[t][3]);
    // dh -= dv^T w
#pragma unroll
    for (int i = 0; i < 4; ++i) split_acc(dv[2 * i], dv[2 * i + 1], af[i]);
#pragma unroll
    for (int cp = 0; cp < KT; cp += CW) {
      float sub[2 * CW][4];
      chunk_sum<CW>(sub, af, [&](int i, int x) { return ld_b_t(st + St::w, pair_at(i) * 16, kq * KT + cp + x, L); });
#pragma unroll
      for (int t = 0; t < 2 * CW; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) dh[2 * cp + t][e] -= sub[t][e];
    }
    __syncwarp();
    if (lane == 0) ptx::mbar_arrive(empty_bar(s));
  }
  if (a.dh0 != nullptr && live && ok) {
#pragma unroll
    for (int t = 0; t < 2 * KT; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int kk = k0 + t * 8 + kc + (e & 1), vv = vr + (e >> 1) * 8;
        if (kk < D.K && vv < D.V) a.dh0[hbase + (long long)kk * D.V + vv] = dh[t][e];
      }
  }
  __syncthreads();
}

// Both scans of the backward pass: neither reads what the other writes.  CTAs below `nx` walk the sequence backwards, the others
// forwards again.  A scan is a chain over the chunks, so running them side by side takes the longer one's time where the SMs
// hold both (whole backward pass at K = V = 128: B=1, S=8192, H=4 587 -> 396 us; B=1, S=4096, H=8 373 -> 275 us; B=2, S=4096, H=8
// 485 -> 443 us).  Where they do not, one launch each: mixed, B=8, S=4096, H=8 took 1564 us instead of 1488.
// SIDE: 0 the two by blockIdx, 1 the forward scan alone, 2 the reverse scan alone.
template <int KB, int NG, int KS, int SIDE>
__global__ void __launch_bounds__(scan_threads(NG * KS), 1)
bwd_scans_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_at, const __grid_constant__ CUtensorMap tm_do, const ScanArgs fwd, const RevArgs rev,
                 int nx) {
  if (SIDE == 2 || (SIDE == 0 && (int)blockIdx.x < nx))
    rev_scan<KB, NG, KS>(tm_w, tm_q, tm_k, tm_at, tm_do, rev, blockIdx.x);
  else
    fwd_scan<KB, NG, KS, true>(tm_w, tm_q, tm_k, tm_at, fwd, SIDE == 1 ? (int)blockIdx.x : (int)blockIdx.x - nx);
}

// ------------------------------------------------------------------------------------------------ chunk kernel

constexpr int kBwdThreads = 512;
constexpr int kVBox = 16 * 128;      // a [16 rows][64 bf16] tile

// Shared memory: tiles k, q*scale, k*beta, v*beta, do; the pieces of A; the pieces of dvb (later those of T and dP); the stage
// (two buffers for 16 columns of V each: pieces of h_in, dh, v_new; before that S, A and scratch in float32; later the pieces of dkg, then
// those of X); gates, beta and the partial sums.
struct BwdSmem {
  int k, q, kb, vb, d_o, a, dvb, t, dp, stage, sh, sdh, svn, vbuf, gates, beta, red, total;
};
__host__ __device__ constexpr BwdSmem bwd_smem(int kboxes, int vboxes) {
  BwdSmem m{};
  m.k = 0;
  m.q = kboxes * kBox;
  m.kb = 2 * kboxes * kBox;
  m.vb = 3 * kboxes * kBox;
  m.d_o = m.vb + vboxes * kBox;
  m.a = m.d_o + vboxes * kBox;
  m.dvb = m.a + 3 * kBox;
  m.t = m.dvb;
  m.dp = m.dvb + 3 * kBox;
  m.stage = m.dvb + 6 * kBox;
  m.sh = 0;   // within one of the two buffers of the stage
  m.sdh = m.sh + 3 * kboxes * kVBox;
  m.svn = m.sdh + 3 * kboxes * kVBox;
  m.vbuf = m.svn + 3 * kVBox;
  const int stage_end = m.stage + 2 * m.vbuf, scratch_end = m.stage + (2 * C + 32) * kSP * 4;
  m.gates = stage_end > scratch_end ? stage_end : scratch_end;
  m.beta = m.gates + kGateBytes;
  m.red = m.beta + C * 4;
  m.total = m.red + 28 * C * 4 + 64;
  return m;
}

struct BwdArgs {
  const __nv_bfloat16 *k, *v, *beta, *d_o;
  const uint8_t *fws, *bws;
  __nv_bfloat16 *dq, *dk, *dv, *dbeta;
  float* dg;
  Dims D;
};

// two adjacent floats -> their three pieces at (row, col) of a swizzled tile whose pieces are `piece_stride` bytes apart
__device__ __forceinline__ void put_pieces(uint32_t tile, int piece_stride, int row, int col, float x0, float x1) {
  uint32_t p0, p1, p2;
  split3(x0, x1, p0, p1, p2);
  const uint32_t at = swz(tile, row, col >> 3) + (col & 7) * 2;
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(p0) : "memory");
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + piece_stride), "r"(p1) : "memory");
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(at + 2 * piece_stride), "r"(p2) : "memory");
}
__device__ __forceinline__ uint32_t ld_shared32(uint32_t at) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
  return v;
}
// ANY: at any address of the element type (an instance of its own: the choice inside the kernel took 2 % of its time)
template <bool ANY>
__device__ __forceinline__ void st_pair(__nv_bfloat16* p, uint32_t v) {
  if constexpr (ANY) {
    reinterpret_cast<uint16_t*>(p)[0] = (uint16_t)v;
    reinterpret_cast<uint16_t*>(p)[1] = (uint16_t)(v >> 16);
  } else {
    *reinterpret_cast<uint32_t*>(p) = v;
  }
}
__device__ __forceinline__ float quad_sum(float v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// One CTA of 16 warps per chunk and head.  [64, K] results: warp (wm, wc) owns 16 tokens and a quarter of the columns;
// [64, 64] results: one 16 x 16 tile.  What contracts over V (dqE, dkg, dkd, dattn: 8,000 of the 12,600 MMAs at K = V = 128)
// runs over 16 columns at a time, whose pieces of h_in, dh and v_new all warps cut and share.
// dqE, dkg and dkd are summed up by the tensor core: they leave in bf16, and dg, which takes their row sums, is no further from 64 bits
// for it (2.3e-7 of its norm at 512 tokens, K = V = 128; 3.8e-7 in float32 on the CUDA cores; summed up with rounding 1.9e-7, and
// this kernel 1.10 ms).  The [64, 64] sums, whose results are cut into pieces again, are rounded (gdn_mma.cuh).
// B=8, S=4096, H=8, K=V=128: 0.96 ms (4.43 ms in float32 on the CUDA cores; 1.04 with 32 columns of V between two barriers that all
// cut and then all multiplied, tiles of the [64, 64] matrices by quarters, and loads where they are used).  Of 63,500 cycles a chunk the
// loop over V takes 25,500 for 16,300 of MMAs, dvb 6,600, X 5,500.
template <int KB, int VB, bool ANY>
__global__ void __launch_bounds__(kBwdThreads, 1) bwd_chunk_kernel(const BwdArgs g) {
  extern __shared__ __align__(1024) uint8_t gdn_smem_raw[];
  constexpr BwdSmem M = bwd_smem(KB, VB);
  const uint32_t base = ptx::smem_u32(gdn_smem_raw);
  if ((base & 1023u) != 0) {
    if (threadIdx.x == 0) raise_status(LEWI_STATUS_SMEM_LAYOUT);
    return;
  }
  const uint32_t tK = base + M.k, tQ = base + M.q, tKb = base + M.kb, tVb = base + M.vb, tDo = base + M.d_o, tA = base + M.a,
                 tDvb = base + M.dvb, tT = base + M.t, tDp = base + M.dp, tStage = base + M.stage;
  float* sS = reinterpret_cast<float*>(gdn_smem_raw + M.stage);
  float* sA = sS + C * kSP;
  float* sX = sA + C * kSP;
  float* gates = reinterpret_cast<float*>(gdn_smem_raw + M.gates);
  const float *gcs = gates, *sE = gates + C, *sEk = gates + 2 * C;
  float* sBeta = reinterpret_cast<float*>(gdn_smem_raw + M.beta);
  float* rowG = reinterpret_cast<float*>(gdn_smem_raw + M.red);   // [4][64] each: by tile column / tile row / column quarter
  float* colG = rowG + 4 * C;
  float* rowS = colG + 4 * C;    // rowsum(dqE qE) - rowsum(dkd kd) + rowsum(dkg kg)
  float* rowK = rowS + 4 * C;    // rowsum(dkd kd)
  float* dbK = rowK + 4 * C;     // dbeta, part of dkb
  float* dbV = dbK + 4 * C;      // [8][64] dbeta, part of dvb
  float* sHd = dbV + 8 * C;      // [16] <dh, h_in> by warp
  const int n = blockIdx.x, h = blockIdx.y, b = blockIdx.z;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp & 3, wc = warp >> 2;
  // this warp's 16 x 16 tile of the [64, 64] matrices: the ten that are not above the diagonal come first, which spreads them over the
  // schedulers (3, 3, 2 and 2; by quarters it would be 1, 2, 3 and 4)
  const int tm = (int)(0x940ffa94u >> (2 * warp) & 3), tc = (int)(0xfb9e4910u >> (2 * warp) & 3);
  const bool active = tc <= tm;
  const int er = lane >> 2, ec = (lane & 3) * 2;      // this lane's elements of an accumulator tile
  const LaneOff L = lane_off(lane);
  const Dims& D = g.D;
  const int K = D.K, V = D.V;
  const long long chunk = ((long long)b * D.N + n) * D.H + h, tok0 = (long long)n * C;
  const FwdWs FW = fwd_ws(D);
  const BwdWs BW = bwd_ws(D);
  const float scale = round_bf16(rsqrtf((float)K));
  auto row_off = [&](int r) { return ((long long)b * D.S + tok0 + r) * D.H + h; };
  auto in_seq = [&](int r) { return tok0 + r < D.S; };

  // ---- loads (all requested before any is used); rows past the end of the sequence are zero
  {
    const __nv_bfloat16* qs = reinterpret_cast<const __nv_bfloat16*>(g.fws + FW.qs) + chunk * C * K;
    uint4 kr[KB], qr[KB], vr[VB], dr[VB];
    __nv_bfloat16 bk[KB], bv[VB];
    const uint4 zero = make_uint4(0, 0, 0, 0);
    const __nv_bfloat16 bzero = __float2bfloat16_rn(0.f);
#pragma unroll
    for (int x = 0; x < KB; ++x) {
      const int i = x * kBwdThreads + tid, r = i / (KB * 8), p = i % (KB * 8);
      const bool in = in_seq(r) && p * 8 < K;
      kr[x] = in ? ld_nc_v4(g.k + row_off(r) * K + p * 8) : zero;
      qr[x] = in ? ld_nc_v4(qs + r * K + p * 8) : zero;
      bk[x] = in ? g.beta[row_off(r)] : bzero;
    }
#pragma unroll
    for (int x = 0; x < VB; ++x) {
      const int i = x * kBwdThreads + tid, r = i / (VB * 8), p = i % (VB * 8);
      const bool in = in_seq(r) && p * 8 < V;
      vr[x] = in ? ld_nc_v4(g.v + row_off(r) * V + p * 8) : zero;
      dr[x] = in ? ld_nc_v4(g.d_o + row_off(r) * V + p * 8) : zero;
      bv[x] = in ? g.beta[row_off(r)] : bzero;
    }
    if (tid < 3 * C) gates[tid] = reinterpret_cast<const float*>(g.fws + FW.gates)[chunk * 3 * C + tid];
    if (tid < C) sBeta[tid] = in_seq(tid) ? __bfloat162float(g.beta[row_off(tid)]) : 0.f;
#pragma unroll
    for (int x = 0; x < KB; ++x) {
      const int i = x * kBwdThreads + tid, r = i / (KB * 8), p = i % (KB * 8);
      const uint32_t at = swz((p >> 3) * kBox, r, p & 7);
      st_shared16(tK + at, kr[x]);
      st_shared16(tQ + at, qr[x]);
      st_shared16(tKb + at, scaled_piece(kr[x], bk[x]));
    }
#pragma unroll
    for (int x = 0; x < VB; ++x) {
      const int i = x * kBwdThreads + tid, r = i / (VB * 8), p = i % (VB * 8);
      const uint32_t at = swz((p >> 3) * kBox, r, p & 7);
      st_shared16(tVb + at, scaled_piece(vr[x], bv[x]));
      st_shared16(tDo + at, dr[x]);
    }
  }
  __syncthreads();

  // dv_new of this warp's 16 columns of V (see below), requested long before it is used
  const int nvb = (BW.v16 + 1) / 2, dblk = warp >> 1;   // blocks of 32 columns of V; the warp's block of 16
  float4 dvt[8];
  {
    const float4* src = reinterpret_cast<const float4*>(g.bws + BW.dv) + (chunk * BW.v16 + dblk) * 8 * 32 + lane;
#pragma unroll
    for (int t = 0; t < 8; ++t) dvt[t] = dblk < BW.v16 ? src[t * 32] : make_float4(0.f, 0.f, 0.f, 0.f);
  }

  // ---- bf16(kb k^T) and P = bf16(q k^T), kept as packed bf16; S to shared memory
  uint32_t ps[4] = {0, 0, 0, 0}, pa[4] = {0, 0, 0, 0};
  auto decay = [&](int r, int c) { return __expf(gcs[r] - gcs[c]); };
  if (active) {
    float s2[2][4], a2[2][4];
    zero4(s2[0]); zero4(s2[1]); zero4(a2[0]); zero4(a2[1]);
#pragma unroll
    for (int ks = 0; ks < 4 * KB; ++ks) {
      const Frag4 bb = ld_b(tK, tc * 16, ks, L);
      mma2_add(s2[0], s2[1], ld_a(tKb, tm * 16, ks, L).r, bb);
      mma2_add(a2[0], a2[1], ld_a(tQ, tm * 16, ks, L).r, bb);
    }
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        ps[t * 2 + e] = pack_bf16(s2[t][2 * e], s2[t][2 * e + 1]);
        pa[t * 2 + e] = pack_bf16(a2[t][2 * e], a2[t][2 * e + 1]);
        const int r = tm * 16 + er + 8 * e, c = tc * 16 + t * 8 + ec;
        *reinterpret_cast<float2*>(sS + r * kSP + c) =
            make_float2(c < r ? bf16_lo(ps[t * 2 + e]) * decay(r, c) : 0.f, c + 1 < r ? bf16_hi(ps[t * 2 + e]) * decay(r, c + 1) : 0.f);
      }
  }
  __syncthreads();
  unit_lower_inverse(sS, sA, sX, tid);
  {   // the pieces of A
    const int r = tid >> 3, p = tid & 7;
    const float4 lo = *reinterpret_cast<const float4*>(sA + r * kSP + p * 8), hi = *reinterpret_cast<const float4*>(sA + r * kSP + p * 8 + 4);
    const float a[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
    uint32_t pc[3][4];
#pragma unroll
    for (int x = 0; x < 4; ++x) split3(a[2 * x], a[2 * x + 1], pc[0][x], pc[1][x], pc[2][x]);
#pragma unroll
    for (int w3 = 0; w3 < 3; ++w3) st_shared16(swz(tA + w3 * kBox, r, p), make_uint4(pc[w3][0], pc[w3][1], pc[w3][2], pc[w3][3]));
  }
  __syncthreads();

  // ---- dvb = A^T dv_new: warp = (16 columns of V, 32 of the tokens); its pieces to shared memory, dv, part of dbeta
  // what the first pass over V needs is requested here
  const float4* hs_in = reinterpret_cast<const float4*>(g.bws + BW.hs) + chunk * BW.v16 * (8 * KB) * 32 + warp * 32 + lane;
  const float4* dh_in = reinterpret_cast<const float4*>(g.bws + BW.dh) + chunk * BW.v16 * (8 * KB) * 32 + warp * 32 + lane;
  const float4* vn_in = reinterpret_cast<const float4*>(g.bws + BW.vn) + chunk * BW.v16 * 8 * 32 + warp * 32 + lane;
  float4 hr, dr, vr;   // this warp's tile of h_in^T, dh^T and (the first eight warps) v_new^T
  auto fetch = [&](int vb) {
    if (warp < 8 * KB) {
      hr = hs_in[vb * (8 * KB) * 32];
      dr = dh_in[vb * (8 * KB) * 32];
    }
    if (warp < 8) vr = vn_in[vb * 8 * 32];
  };
  fetch(0);
  {
    const int blk = dblk;
    if (blk < 2 * nvb) {
      // token blocks 0, 3 or 1, 2 (A^T is upper triangular: the sum of block m runs over m..3)
      const int mrow[2] = {warp & 1, 3 - (warp & 1)};
      uint32_t vv[2][2][2];
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int r = mrow[x] * 16 + er + 8 * e, c = blk * 16 + t * 8 + ec;
            vv[x][e][t] = in_seq(r) && c < V ? *reinterpret_cast<const uint32_t*>(g.v + row_off(r) * V + c) : 0u;
          }
      float acc[2][2][4];
#pragma unroll
      for (int x = 0; x < 2; ++x) { zero4(acc[x][0]); zero4(acc[x][1]); }
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        uint32_t b0[3][2], b1[3][2];   // an accumulator tile of dv^T is the B operand of this product
        split3(dvt[2 * ks].x, dvt[2 * ks].y, b0[0][0], b0[1][0], b0[2][0]);
        split3(dvt[2 * ks + 1].x, dvt[2 * ks + 1].y, b0[0][1], b0[1][1], b0[2][1]);
        split3(dvt[2 * ks].z, dvt[2 * ks].w, b1[0][0], b1[1][0], b1[2][0]);
        split3(dvt[2 * ks + 1].z, dvt[2 * ks + 1].w, b1[0][1], b1[1][1], b1[2][1]);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          if (ks < mrow[x]) continue;
          const Frag3x4 fa = ld_a3_t(tA, kBox, ks * 16, mrow[x], L);
          mma_x6(acc[x][0], fa, b0);
          mma_x6(acc[x][1], fa, b1);
        }
      }
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int r = mrow[x] * 16 + er + 8 * e;
          const float be = sBeta[r];
          float rb = 0.f;
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            const int c = blk * 16 + t * 8 + ec;
            const float d0 = acc[x][t][2 * e], d1 = acc[x][t][2 * e + 1];
            put_pieces(tDvb + (c >> 6) * kBox, VB * kBox, r, c & 63, d0, d1);
            if (in_seq(r) && c < V) {
              rb = fmaf(d0, bf16_lo(vv[x][e][t]), rb);
              rb = fmaf(d1, bf16_hi(vv[x][e][t]), rb);
              st_pair<ANY>(g.dv + row_off(r) * V + c, pack_bf16(d0 * be, d1 * be));
            }
          }
          rb = quad_sum(rb);
          if ((lane & 3) == 0) dbV[blk * C + r] = rb;
        }
    }
  }

  // ---- over V, 16 columns at a time: dqE = do h_in^T, -dkg = dvb h_in^T, dkd = v_new dh^T, dattn = do v_new^T.  Two buffers: while a
  // block is multiplied the pieces of the next one are cut into the other, and the one after that is on its way from memory.
  float dq[2 * KB][4], dkb[2 * KB][4], dk[2 * KB][4], dat[2][4];
#pragma unroll
  for (int t = 0; t < 2 * KB; ++t) { zero4(dq[t]); zero4(dkb[t]); zero4(dk[t]); }
  zero4(dat[0]); zero4(dat[1]);
  float hd = 0.f;                                     // <dh, h_in>
  {
    auto put = [&](int vb) {
      const uint32_t buf = tStage + (vb & 1) * M.vbuf;
      const int c = (warp & 7) * 8 + ec;
      if (warp < 8 * KB) {
        const uint32_t box = (warp >> 3) * kVBox;
        put_pieces(buf + M.sh + box, KB * kVBox, er, c, hr.x, hr.y);
        put_pieces(buf + M.sh + box, KB * kVBox, er + 8, c, hr.z, hr.w);
        put_pieces(buf + M.sdh + box, KB * kVBox, er, c, dr.x, dr.y);
        put_pieces(buf + M.sdh + box, KB * kVBox, er + 8, c, dr.z, dr.w);
        hd = fmaf(hr.x, dr.x, hd); hd = fmaf(hr.y, dr.y, hd);
        hd = fmaf(hr.z, dr.z, hd); hd = fmaf(hr.w, dr.w, hd);
      }
      if (warp < 8) {
        put_pieces(buf + M.svn, kVBox, er, c, vr.x, vr.y);
        put_pieces(buf + M.svn, kVBox, er + 8, c, vr.z, vr.w);
      }
    };
    __syncthreads();   // the float32 scratch is dead
    put(0);
    if (BW.v16 > 1) fetch(1);
    __syncthreads();   // (the pieces of dvb are complete, too)
    for (int ks = 0; ks < BW.v16; ++ks) {
      const uint32_t buf = tStage + (ks & 1) * M.vbuf;
      if (ks + 1 < BW.v16) put(ks + 1);
      if (ks + 2 < BW.v16) fetch(ks + 2);
      const Frag4 fdo = ld_a(tDo, wm * 16, ks, L);
      const Frag3x4 fdvb = ld_a3(tDvb, VB * kBox, wm * 16, ks, L), fvn = ld_a3_t(buf + M.svn, kVBox, 0, wm, L);
#pragma unroll
      for (int cp = 0; cp < KB; ++cp) {
        const int np = wc * KB + cp;
        Frag4 hb[3];
#pragma unroll
        for (int w3 = 0; w3 < 3; ++w3) hb[w3] = ld_b_t(buf + M.sh + w3 * KB * kVBox, 0, np, L, kVBox);
        mma2(dq[2 * cp], dq[2 * cp + 1], fdo.r, hb[2]);
        mma2_x6_acc(dkb[2 * cp], dkb[2 * cp + 1], fdvb, hb);
        mma2(dq[2 * cp], dq[2 * cp + 1], fdo.r, hb[1]);
        mma2(dq[2 * cp], dq[2 * cp + 1], fdo.r, hb[0]);
#pragma unroll
        for (int w3 = 0; w3 < 3; ++w3) hb[w3] = ld_b_t(buf + M.sdh + w3 * KB * kVBox, 0, np, L, kVBox);
        mma2_x6_acc(dk[2 * cp], dk[2 * cp + 1], fvn, hb);
      }
      if (active) {
        const Frag4 b[3] = {ld_b_t(buf + M.svn, 0, tc, L), ld_b_t(buf + M.svn + kVBox, 0, tc, L), ld_b_t(buf + M.svn + 2 * kVBox, 0, tc, L)};
        mma2_x3(dat[0], dat[1], ld_a(tDo, tm * 16, ks, L).r, b);
      }
      __syncthreads();
    }
  }
  hd = warp_sum(hd);
  if (lane == 0) sHd[warp] = hd;

  // ---- row sums, the decays of the rows, the pieces of dkg (everybody is done with the stage)
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int r = wm * 16 + er + 8 * e;
    const float ee = sE[r], ek = sEk[r];
    float sq = 0.f, sk = 0.f, sg = 0.f;
#pragma unroll
    for (int t = 0; t < 2 * KB; ++t) {
      const int c = wc * 16 * KB + t * 8 + ec;
      const uint32_t at = swz((c >> 6) * kBox, r, (c & 63) >> 3) + (c & 7) * 2;
      const uint32_t qq = ld_shared32(tQ + at), kk = ld_shared32(tK + at), kbv = ld_shared32(tKb + at);
      const float g0 = -dkb[t][2 * e], g1 = -dkb[t][2 * e + 1];
      sq = fmaf(dq[t][2 * e], bf16_lo(qq), sq); sq = fmaf(dq[t][2 * e + 1], bf16_hi(qq), sq);
      sk = fmaf(dk[t][2 * e], bf16_lo(kk), sk); sk = fmaf(dk[t][2 * e + 1], bf16_hi(kk), sk);
      sg = fmaf(g0, bf16_lo(kbv), sg); sg = fmaf(g1, bf16_hi(kbv), sg);
      put_pieces(tStage + (c >> 6) * kBox, KB * kBox, r, c & 63, g0, g1);
      dkb[t][2 * e] = g0 * ee; dkb[t][2 * e + 1] = g1 * ee;
      dq[t][2 * e] *= ee; dq[t][2 * e + 1] *= ee;
      dk[t][2 * e] *= ek; dk[t][2 * e + 1] *= ek;
    }
    sq = quad_sum(sq); sk = quad_sum(sk); sg = quad_sum(sg);
    if ((lane & 3) == 0) {
      rowS[wc * C + r] = ee * (sq + sg) - ek * sk;
      rowK[wc * C + r] = ek * sk;
    }
  }
  __syncthreads();

  // ---- X = dvb vb^T + dkg kg^T (this warp's tile)
  float x1[2][4], x2[2][4];
  zero4(x1[0]); zero4(x1[1]); zero4(x2[0]); zero4(x2[1]);
  if (active) {
    for (int ks = 0; ks < 2 * nvb; ++ks) {
      const Frag4 bb = ld_b(tVb, tc * 16, ks, L);
      mma2_x3(x1[0], x1[1], ld_a3(tDvb, VB * kBox, tm * 16, ks, L), bb);
    }
#pragma unroll
    for (int ks = 0; ks < 4 * KB; ++ks) {
      const Frag4 bb = ld_b(tKb, tc * 16, ks, L);
      mma2_x3(x2[0], x2[1], ld_a3(tStage, KB * kBox, tm * 16, ks, L), bb);
    }
  }
  __syncthreads();   // dvb and dkg have been read: their places take T and X
  float gg[2][4];
  zero4(gg[0]); zero4(gg[1]);
  if (active) {
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = tm * 16 + er + 8 * e, c = tc * 16 + t * 8 + ec;
        put_pieces(tStage, kBox, r, c, fmaf(x2[t][2 * e], sE[c], x1[t][2 * e]), fmaf(x2[t][2 * e + 1], sE[c + 1], x1[t][2 * e + 1]));
        const float t0 = c <= r ? dat[t][2 * e] * decay(r, c) : 0.f, t1 = c + 1 <= r ? dat[t][2 * e + 1] * decay(r, c + 1) : 0.f;
        put_pieces(tT, kBox, r, c, t0, t1);
        gg[t][2 * e] = t0 * bf16_lo(pa[t * 2 + e]);
        gg[t][2 * e + 1] = t1 * bf16_hi(pa[t * 2 + e]);
      }
  }
  __syncthreads();

  // ---- dS = -strict(X A^T), dP = dS D, G = T P + dS S
  float ds[2][4];
  zero4(ds[0]); zero4(ds[1]);
  if (active) {
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      if (ks > tc) break;
      const Frag4 b[3] = {ld_b(tA, tc * 16, ks, L), ld_b(tA + kBox, tc * 16, ks, L), ld_b(tA + 2 * kBox, tc * 16, ks, L)};
      mma2_x6(ds[0], ds[1], ld_a3(tStage, kBox, tm * 16, ks, L), b);
    }
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = tm * 16 + er + 8 * e, c = tc * 16 + t * 8 + ec;
        const float p0 = c < r ? -ds[t][2 * e] * decay(r, c) : 0.f, p1 = c + 1 < r ? -ds[t][2 * e + 1] * decay(r, c + 1) : 0.f;
        put_pieces(tDp, kBox, r, c, p0, p1);
        gg[t][2 * e] = fmaf(p0, bf16_lo(ps[t * 2 + e]), gg[t][2 * e]);      // dS S = dP bf16(kb k^T)
        gg[t][2 * e + 1] = fmaf(p1, bf16_hi(ps[t * 2 + e]), gg[t][2 * e + 1]);
      }
  }
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const float rs = quad_sum(gg[0][2 * e] + gg[0][2 * e + 1] + gg[1][2 * e] + gg[1][2 * e + 1]);
    if ((lane & 3) == 0) rowG[tc * C + tm * 16 + er + 8 * e] = rs;
  }
#pragma unroll
  for (int t = 0; t < 2; ++t)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float cs = gg[t][e] + gg[t][2 + e];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) cs += __shfl_xor_sync(0xffffffffu, cs, o);
      if (lane < 4) colG[tm * C + tc * 16 + t * 8 + ec + e] = cs;
    }

  // ---- dq += T k, dk += T^T q (rounded to bf16 next: accumulated by the tensor core, like dkb and dk below)
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
    for (int cp = 0; cp < KB; ++cp) {
      const int np = wc * KB + cp;
      if (ks <= wm) {
        const Frag4 bb = ld_b_t(tK, ks * 16, np, L);
#pragma unroll
        for (int w3 = 2; w3 >= 0; --w3) mma2(dq[2 * cp], dq[2 * cp + 1], ld_a(tT + w3 * kBox, wm * 16, ks, L).r, bb);
      }
      if (ks >= wm) {
        const Frag4 bb = ld_b_t(tQ, ks * 16, np, L);
#pragma unroll
        for (int w3 = 2; w3 >= 0; --w3) mma2(dk[2 * cp], dk[2 * cp + 1], ld_a_t(tT + w3 * kBox, ks * 16, wm, L).r, bb);
      }
    }
  }
#pragma unroll
  for (int t = 0; t < 2 * KB; ++t)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = wm * 16 + er + 8 * e, c = wc * 16 * KB + t * 8 + ec;
      if (in_seq(r) && c < K) st_pair<ANY>(g.dq + row_off(r) * K + c, pack_bf16(dq[t][2 * e] * scale, dq[t][2 * e + 1] * scale));
    }
  __syncthreads();

  // ---- dkb += dP k, dk += dP^T kb + dkb beta, part of dbeta
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) {
#pragma unroll
    for (int cp = 0; cp < KB; ++cp) {
      const int np = wc * KB + cp;
      if (ks <= wm) {
        const Frag4 bb = ld_b_t(tK, ks * 16, np, L);
#pragma unroll
        for (int w3 = 2; w3 >= 0; --w3) mma2(dkb[2 * cp], dkb[2 * cp + 1], ld_a(tDp + w3 * kBox, wm * 16, ks, L).r, bb);
      }
      if (ks >= wm) {
        const Frag4 bb = ld_b_t(tKb, ks * 16, np, L);
#pragma unroll
        for (int w3 = 2; w3 >= 0; --w3) mma2(dk[2 * cp], dk[2 * cp + 1], ld_a_t(tDp + w3 * kBox, ks * 16, wm, L).r, bb);
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int r = wm * 16 + er + 8 * e;
    const float be = sBeta[r];
    float rb = 0.f;
#pragma unroll
    for (int t = 0; t < 2 * KB; ++t) {
      const int c = wc * 16 * KB + t * 8 + ec;
      const uint32_t kk = ld_shared32(swz(tK + (c >> 6) * kBox, r, (c & 63) >> 3) + (c & 7) * 2);
      rb = fmaf(dkb[t][2 * e], bf16_lo(kk), rb);
      rb = fmaf(dkb[t][2 * e + 1], bf16_hi(kk), rb);
      if (in_seq(r) && c < K)
        st_pair<ANY>(g.dk + row_off(r) * K + c, pack_bf16(fmaf(dkb[t][2 * e], be, dk[t][2 * e]), fmaf(dkb[t][2 * e + 1], be, dk[t][2 * e + 1])));
    }
    rb = quad_sum(rb);
    if ((lane & 3) == 0) dbK[wc * C + r] = rb;
  }
  __syncthreads();

  // ---- dg = reverse cumulative sum of dgcs, dbeta: warp 0, two tokens per lane
  if (warp == 0) {
    float x[2], rk = 0.f;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = 2 * lane + e;
      float s = 0.f;
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        s += rowG[y * C + r] - colG[y * C + r] + rowS[y * C + r];
        rk += rowK[y * C + r];
      }
      x[e] = s;
      float db = dbK[r] + dbK[C + r] + dbK[2 * C + r] + dbK[3 * C + r];
      for (int y = 0; y < BW.v16; ++y) db += dbV[y * C + r];
      if (in_seq(r)) g.dbeta[row_off(r)] = __float2bfloat16_rn(db);
    }
    const float all = warp_sum(rk) + sE[C - 1] * warp_sum(lane < 16 ? sHd[lane] : 0.f);
    if (lane == 31) x[1] += all;
    float run = x[0] + x[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float up = __shfl_down_sync(0xffffffffu, run, o);
      if (lane + o < 32) run += up;
    }
    const float after = __shfl_down_sync(0xffffffffu, run, 1);
    const float d1 = (lane < 31 ? after : 0.f) + x[1];
    if (in_seq(2 * lane + 1)) g.dg[row_off(2 * lane + 1)] = d1;
    if (in_seq(2 * lane)) g.dg[row_off(2 * lane)] = d1 + x[0];
  }
}

// ------------------------------------------------------------------------------------------------ host side

struct RevMaps {
  CUtensorMap w, q, k, at, d_o;
};

template <int KB, int NG, int KS, int SIDE>
inline int launch_scans_side(cudaStream_t st, const RevMaps& m, const ScanArgs& fwd, const RevArgs& rev) {
  static bool done[64] = {false};
  constexpr int smem_f = ScanSmem<KB, NG, KS>::total, smem_r = RevSmem<KB, NG, KS>::total;
  constexpr int smem = SIDE == 1 ? smem_f : (SIDE == 2 ? smem_r : (smem_r > smem_f ? smem_r : smem_f));
  if (!allow_smem(bwd_scans_kernel<KB, NG, KS, SIDE>, smem, done)) return LEWI_ERR_CUDA;
  const int nx = (rev.v16 + NG - 1) / NG;
  bwd_scans_kernel<KB, NG, KS, SIDE><<<dim3((unsigned)(SIDE == 0 ? 2 * nx : nx), (unsigned)rev.D.H, (unsigned)rev.D.B), scan_threads(NG * KS), smem,
                                       st>>>(m.w, m.q, m.k, m.at, m.d_o, fwd, rev, nx);
  LEWI_CHECK_LAUNCH();
  return LEWI_OK;
}
template <int KB, int NG, int KS>
inline int launch_scans(cudaStream_t st, const RevMaps& m, const ScanArgs& fwd, const RevArgs& rev, bool together) {
  if constexpr (NG <= 2) {   // (four or eight groups are taken where twice as many CTAs do not fit)
    if (together) return launch_scans_side<KB, NG, KS, 0>(st, m, fwd, rev);
  }
  if (int rc = launch_scans_side<KB, NG, KS, 1>(st, m, fwd, rev)) return rc;
  return launch_scans_side<KB, NG, KS, 2>(st, m, fwd, rev);
}

template <int KB, int VB, bool ANY>
inline int launch_bwd_chunk(cudaStream_t st, const BwdArgs& a) {
  static bool done[64] = {false};
  constexpr int smem = bwd_smem(KB, VB).total;
  static_assert(smem <= 227 * 1024, "shared memory of the chunk kernel");
  if (!allow_smem(bwd_chunk_kernel<KB, VB, ANY>, smem, done)) return LEWI_ERR_CUDA;
  bwd_chunk_kernel<KB, VB, ANY><<<dim3((unsigned)a.D.N, (unsigned)a.D.H, (unsigned)a.D.B), kBwdThreads, smem, st>>>(a);
  LEWI_CHECK_LAUNCH();
  return LEWI_OK;
}

template <int KB>
inline int backward(cudaStream_t st, const void* k, const void* v, const void* beta, const float* h0, const void* d_o,
                    const float* dh_final, const uint8_t* fws, uint8_t* bws, void* dq, void* dk, void* dv, float* dg, void* dbeta,
                    float* dh0, const Dims& D) {
  const FwdWs FW = fwd_ws(D);
  const BwdWs BW = bwd_ws(D);
  if ((reinterpret_cast<uintptr_t>(d_o) & 15u) != 0) {
    if (cudaMemcpyAsync(bws + BW.d_o, d_o, (size_t)D.B * D.S * D.H * D.V * 2, cudaMemcpyDeviceToDevice, st) != cudaSuccess) {
      (void)cudaGetLastError();
      return LEWI_ERR_CUDA;
    }
    d_o = bws + BW.d_o;
  }
  const float* gates = reinterpret_cast<const float*>(fws + FW.gates);
  const ScanArgs sa{reinterpret_cast<const uint32_t*>(fws + FW.ut), gates, h0, nullptr, nullptr, reinterpret_cast<float4*>(bws + BW.hs),
                    reinterpret_cast<float4*>(bws + BW.vn), FW.v16, D};
  const long long rows = (long long)D.B * D.N * D.H * C;
  RevMaps m;
  if (!rows_map(&m.w, fws + FW.w, D.K, rows, C) || !rows_map(&m.q, fws + FW.qs, D.K, rows, C) || !heads_map(&m.k, k, D.B, D.S, D.H, D.K) ||
      !rows_map(&m.at, fws + FW.attn, C, 3 * rows, 3 * C) || !heads_map(&m.d_o, d_o, D.B, D.S, D.H, D.V))
    return LEWI_ERR_CUDA;
  const RevArgs ra{gates, dh_final, dh0, reinterpret_cast<float4*>(bws + BW.dh), reinterpret_cast<float4*>(bws + BW.dv), FW.v16, D};
  // groups per CTA as in the forward pass, or two instead of one where that makes room for both scans (a warp's work is the same)
  int ng = scan_groups(D, FW.v16), rc;
  auto both_fit = [&](int groups) { return 2ll * D.B * D.H * ((FW.v16 + groups - 1) / groups) <= num_sms(); };
  bool together = both_fit(ng);
  if (!together && ng == 1 && both_fit(2)) {
    ng = 2;
    together = true;
  }
  switch (ng) {
    case 1: rc = launch_scans<KB, 1, 4>(st, m, sa, ra, together); break;
    case 2: rc = launch_scans<KB, 2, 4>(st, m, sa, ra, together); break;
    case 4: rc = launch_scans<KB, 4, 2>(st, m, sa, ra, together); break;
    default: rc = launch_scans<KB, 8, 1>(st, m, sa, ra, together); break;
  }
  if (rc) return rc;
  using bf = __nv_bfloat16;
  const BwdArgs ba{reinterpret_cast<const bf*>(k), reinterpret_cast<const bf*>(v), reinterpret_cast<const bf*>(beta), reinterpret_cast<const bf*>(d_o),
                   fws, bws, reinterpret_cast<bf*>(dq), reinterpret_cast<bf*>(dk), reinterpret_cast<bf*>(dv), reinterpret_cast<bf*>(dbeta), dg, D};
  const bool any = ((reinterpret_cast<uintptr_t>(dq) | reinterpret_cast<uintptr_t>(dk) | reinterpret_cast<uintptr_t>(dv)) & 3u) != 0;
  if (D.V <= 64) return any ? launch_bwd_chunk<KB, 1, true>(st, ba) : launch_bwd_chunk<KB, 1, false>(st, ba);
  return any ? launch_bwd_chunk<KB, 2, true>(st, ba) : launch_bwd_chunk<KB, 2, false>(st, ba);
}

}  // namespace gdn
}  // namespace lewi
