// Warp-level tensor-core pieces of the gated delta rule kernels (gdn_fwd.cuh, gdn_bwd.cuh).
//
// The recurrence multiplies a float32 state, held in registers as the accumulator of one product, into the next one.
// `mma.sync` (m16n8k16, bf16 in, f32 accumulate) takes that operand from registers: the accumulator layout of two
// 8-column tiles IS the layout of a 16-deep A operand, so a warp carries 16 columns of the state through the whole
// sequence without shared memory or another warp.  (tcgen05 would need the state in tensor memory, a round trip
// tcgen05.ld -> split -> tcgen05.st and two commit waits per 64-token chunk, and 128 state columns per CTA: 64 CTAs at
// batch 8 x 8 heads.)
//
// Float32 operands are cut into three bf16 pieces (8 + 8 + 8 mantissa bits, see split3 for what that excludes), so a product of a
// float32 and a bf16 operand is three MMAs and one of two float32 operands six (piece products below 2^-24 of the whole
// are left out); all of them accumulate in float32, which the tensor core truncates (see Prod2).  Measured on a B200: one
// m16n8k16 per 8 cycles and scheduler.
#pragma once

#include "common.cuh"
#include "tcgen05.cuh"

namespace lewi {
namespace gdn {

constexpr int C = 64;                    // tokens per chunk
constexpr int kMaxK = 128, kMaxV = 512;  // head dimensions
constexpr long long kMaxChunks = 1ll << 23;   // rows of the workspace arrays stay below 2^31
constexpr int kBox = 64 * 128;           // bytes of a [64 rows][64 bf16] tile, 128-byte swizzled

struct Frag4 {
  uint32_t r[4];
};
struct Frag3x4 {   // the three bf16 pieces of a float32 A operand
  uint32_t p[3][4];
};

// 16-byte piece `piece` of row `row` of a 128-byte-swizzled tile (rows of 128 bytes, base 1024-byte aligned)
__device__ __forceinline__ uint32_t swz(uint32_t base, int row, int piece) {
  return base + row * 128 + ((piece ^ (row & 7)) << 4);
}

__device__ __forceinline__ Frag4 ldsm(uint32_t addr) {
  Frag4 f;
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(f.r[0]), "=r"(f.r[1]), "=r"(f.r[2]), "=r"(f.r[3]) : "r"(addr) : "memory");
  return f;
}
__device__ __forceinline__ Frag4 ldsm_t(uint32_t addr) {
  Frag4 f;
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(f.r[0]), "=r"(f.r[1]), "=r"(f.r[2]), "=r"(f.r[3]) : "r"(addr) : "memory");
  return f;
}
__device__ __forceinline__ void stsm_t(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};"
               ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// The four loads of a swizzled tile (x4: 16 rows x 16 columns).  The tile may be several 64-column boxes wide, `stride` bytes
// apart.  What a lane contributes to the address is one of two constants; a step of 16 columns flips bits 5 and 6 of it.
struct LaneOff {
  uint32_t n, t;
};
__device__ __forceinline__ LaneOff lane_off(int lane) {
  return {(((lane & 7) + ((lane >> 4) << 3)) * 128) | ((((lane >> 3) & 1) ^ (lane & 7)) << 4), ((lane & 15) * 128) | (((lane >> 4) ^ (lane & 7)) << 4)};
}
// B operand, source [n][k]: r[0..1] = columns n0..n0+7, r[2..3] = n0+8..n0+15, k = 16*ks ..
__device__ __forceinline__ Frag4 ld_b(uint32_t tile, int n0, int ks, LaneOff L, int stride = kBox) {
  return ldsm(tile + (ks >> 2) * stride + n0 * 128 + (L.n ^ ((ks & 3) << 5)));
}
// B operand, source [k][n]: n = 16*np .., k = k0 .. k0+15
__device__ __forceinline__ Frag4 ld_b_t(uint32_t tile, int k0, int np, LaneOff L, int stride = kBox) {
  return ldsm_t(tile + (np >> 2) * stride + k0 * 128 + (L.t ^ ((np & 3) << 5)));
}
// A operand, source [m][k]: rows m0 .. m0+15, k = 16*ks ..
__device__ __forceinline__ Frag4 ld_a(uint32_t tile, int m0, int ks, LaneOff L, int stride = kBox) {
  return ldsm(tile + (ks >> 2) * stride + m0 * 128 + (L.t ^ ((ks & 3) << 5)));
}
// A operand, source [k][m]: m = 16*mp .., k = k0 .. k0+15
__device__ __forceinline__ Frag4 ld_a_t(uint32_t tile, int k0, int mp, LaneOff L, int stride = kBox) {
  return ldsm_t(tile + (mp >> 2) * stride + k0 * 128 + (L.n ^ ((mp & 3) << 5)));
}

// the three pieces of a float32 A operand, `stride` bytes apart
__device__ __forceinline__ Frag3x4 ld_a3(uint32_t tile, int stride, int m0, int ks, LaneOff L) {
  Frag3x4 f;
#pragma unroll
  for (int w3 = 0; w3 < 3; ++w3) {
    const Frag4 x = ld_a(tile + w3 * stride, m0, ks, L);
#pragma unroll
    for (int e = 0; e < 4; ++e) f.p[w3][e] = x.r[e];
  }
  return f;
}
__device__ __forceinline__ Frag3x4 ld_a3_t(uint32_t tile, int stride, int k0, int mp, LaneOff L) {
  Frag3x4 f;
#pragma unroll
  for (int w3 = 0; w3 < 3; ++w3) {
    const Frag4 x = ld_a_t(tile + w3 * stride, k0, mp, L);
#pragma unroll
    for (int e = 0; e < 4; ++e) f.p[w3][e] = x.r[e];
  }
  return f;
}

__device__ __forceinline__ void zero4(float (&d)[4]) { d[0] = d[1] = d[2] = d[3] = 0.f; }
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// both 8-column tiles of a 16-column B load
__device__ __forceinline__ void mma2(float (&d0)[4], float (&d1)[4], const uint32_t (&a)[4], const Frag4& b) {
  mma(d0, a, b.r[0], b.r[1]);
  mma(d1, a, b.r[2], b.r[3]);
}
// A 16-deep product of both 8-column tiles that is to be added to float32 sums.  The tensor core truncates every sum that it makes
// to float32 (a chain of n instructions comes out short by up to n * 2^-24 of itself, always towards zero), so a product starts
// from zero, its pieces small to large, and is added with one rounding.  Error against 64 bits of the state, its gradient and that of
// g, relative to their norm, where nothing is forgotten over 4096 tokens (K = V = 128): with the state as the accumulator 1.0e-5,
// 9.6e-6, 1.0e-5; so 2.1e-7, 2.0e-7, 2.3e-7; in float32 on the CUDA cores 1.6e-6, 2.0e-7, 3.2e-7.
__device__ __forceinline__ void add4(float (&d)[4], const float (&t)[4]) {   // two at a time, each rounded to nearest
#pragma unroll
  for (int e = 0; e < 4; e += 2)
    asm("{\n\t.reg .b64 p, q;\n\tmov.b64 p, {%0, %1};\n\tmov.b64 q, {%2, %3};\n\tadd.rn.f32x2 p, p, q;\n\tmov.b64 {%0, %1}, p;\n\t}"
        : "+f"(d[e]), "+f"(d[e + 1]) : "f"(t[e]), "f"(t[e + 1]));
}
struct Prod2 {
  float t0[4], t1[4];
  __device__ __forceinline__ Prod2() {
    zero4(t0);
    zero4(t1);
  }
  __device__ __forceinline__ void mul(const uint32_t (&a)[4], const Frag4& b) { mma2(t0, t1, a, b); }
  __device__ __forceinline__ void add_to(float (&d0)[4], float (&d1)[4]) const {
    add4(d0, t0);
    add4(d1, t1);
  }
};
// bf16 A times bf16 B
__device__ __forceinline__ void mma2_add(float (&d0)[4], float (&d1)[4], const uint32_t (&a)[4], const Frag4& b) {
  Prod2 x;
  x.mul(a, b);
  x.add_to(d0, d1);
}
// float32 A (three pieces) times bf16 B
__device__ __forceinline__ void mma2_x3(float (&d0)[4], float (&d1)[4], const Frag3x4& a, const Frag4& b) {
  Prod2 x;
#pragma unroll
  for (int w3 = 2; w3 >= 0; --w3) x.mul(a.p[w3], b);
  x.add_to(d0, d1);
}
// s = the sum over the four 16-deep steps of a chunk of float32 A (steps `a`) times bf16 B (`b(step, x)`: column pair x).  What a
// chunk adds to the state is summed up by itself and then added with one rounding, however many steps it has.
template <int CW, class B>
__device__ __forceinline__ void chunk_sum(float (&s)[2 * CW][4], const Frag3x4 (&a)[4], B b) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    Frag4 bf[CW];
    Prod2 y[CW];
#pragma unroll
    for (int x = 0; x < CW; ++x) bf[x] = b(i, x);
#pragma unroll
    for (int w3 = 2; w3 >= 0; --w3)
#pragma unroll
      for (int x = 0; x < CW; ++x) y[x].mul(a[i].p[w3], bf[x]);
#pragma unroll
    for (int x = 0; x < CW; ++x) {
      if (i == 0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s[2 * x][e] = y[x].t0[e];
          s[2 * x + 1][e] = y[x].t1[e];
        }
      } else {
        y[x].add_to(s[2 * x], s[2 * x + 1]);
      }
    }
  }
}
// bf16 A times float32 B
__device__ __forceinline__ void mma2_x3(float (&d0)[4], float (&d1)[4], const uint32_t (&a)[4], const Frag4 (&b)[3]) {
  Prod2 x;
#pragma unroll
  for (int w3 = 2; w3 >= 0; --w3) x.mul(a, b[w3]);
  x.add_to(d0, d1);
}
// float32 A times float32 B; `_acc`: accumulated by the tensor core, for what is rounded to bf16 next
__device__ __forceinline__ void mma2_x6_acc(float (&d0)[4], float (&d1)[4], const Frag3x4& a, const Frag4 (&b)[3]) {
  mma2(d0, d1, a.p[0], b[2]);
  mma2(d0, d1, a.p[2], b[0]);
  mma2(d0, d1, a.p[1], b[1]);
  mma2(d0, d1, a.p[0], b[1]);
  mma2(d0, d1, a.p[1], b[0]);
  mma2(d0, d1, a.p[0], b[0]);
}
__device__ __forceinline__ void mma2_x6(float (&d0)[4], float (&d1)[4], const Frag3x4& a, const Frag4 (&b)[3]) {
  Prod2 x;
  mma2_x6_acc(x.t0, x.t1, a, b);
  x.add_to(d0, d1);
}

// two floats -> three packed bf16 pairs, x = p0 + p1 + p2 exactly for |x| below bf16's largest value (3.39e38), down to float32
// subnormals.  Larger values, infinities and NaN have NaN among their pieces: what is infinite comes out of a product as NaN.
__device__ __forceinline__ void split3(float x0, float x1, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
  p0 = pack_bf16(x0, x1);
  x0 -= bf16_lo(p0);
  x1 -= bf16_hi(p0);
  p1 = pack_bf16(x0, x1);
  p2 = pack_bf16(x0 - bf16_lo(p1), x1 - bf16_hi(p1));
}
// two adjacent accumulator tiles -> the 16-deep A operand they are
__device__ __forceinline__ void split_acc(const float (&t0)[4], const float (&t1)[4], Frag3x4& f) {
  split3(t0[0], t0[1], f.p[0][0], f.p[1][0], f.p[2][0]);
  split3(t0[2], t0[3], f.p[0][1], f.p[1][1], f.p[2][1]);
  split3(t1[0], t1[1], f.p[0][2], f.p[1][2], f.p[2][2]);
  split3(t1[2], t1[3], f.p[0][3], f.p[1][3], f.p[2][3]);
}

// An output may lie at any address of its element type (2 bytes): whole pieces where its base allows it.
__device__ __forceinline__ void st_out8(__nv_bfloat16* p, uint4 v, const __nv_bfloat16* base) {
  if ((reinterpret_cast<uintptr_t>(base) & 15u) == 0) {
    st_v4(p, v);
    return;
  }
  const uint32_t x[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) reinterpret_cast<uint16_t*>(p)[i] = (uint16_t)(x[i >> 1] >> ((i & 1) * 16));
}
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

struct Dims {
  int B, S, H, K, V, N;   // N = chunks per sequence
};

// What the chunk kernel of the forward pass leaves behind for every chunk, all chunks of one kind in one array
// (chunk = (b*N + n)*H + h), so that a tensor map covers it:
//   qs    bf16 [chunks*64][K]         bf16(q * scale)
//   w     bf16 [chunks*64][K]
//   attn  bf16 [chunks*3*64][64]      the three pieces of the in-chunk attention (blocks above the diagonal are not written)
//   ut    bf16 [chunks][V16][32][32]  u^T as accumulator tiles: lane l of a 16-column block holds, for 8-token tile t and
//                                     half p, the pair u[8t + 2(l%4) + {0,1}][16*blk + l/4 + 8p] at element 4t + 2p
//   gates f32  [chunks][3][64]        gcs, exp(gcs), exp(gcs_last - gcs)
struct FwdWs {
  long long qs, w, attn, ut, gates, total;
  int v16;
};
__host__ __device__ inline FwdWs fwd_ws(const Dims& D) {
  FwdWs o;
  const long long chunks = (long long)D.B * D.N * D.H;
  o.v16 = (D.V + 15) / 16;
  long long run = 0;
  auto take = [&](long long bytes) {
    const long long at = run;
    run += (bytes + 255) / 256 * 256;
    return at;
  };
  o.qs = take(chunks * C * D.K * 2);
  o.w = take(chunks * C * D.K * 2);
  o.attn = take(chunks * 3 * C * C * 2);
  o.ut = take(chunks * o.v16 * 2048);
  o.gates = take(chunks * 3 * C * 4);
  o.total = run;
  return o;
}
constexpr int kGateBytes = 3 * C * 4;

}  // namespace gdn
}  // namespace lewi
