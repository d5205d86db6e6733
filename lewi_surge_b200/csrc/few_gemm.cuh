// Products of few rows with much weight: decode steps, short prompts, and the router projection of both.
//
// What bounds them is the weights' way from HBM, once each, so the operands change places against grouped_gemm.cuh: 128 weight
// columns are the M of the MMA (MN-major, as they lie in memory) and a block's rows its N, as many as the block has, rounded up to 16.
// A contraction step then brings 16 KB of weights and 128 bytes per row, where the 256 x 256 tiles of a CTA pair bring 16 KB of rows
// (mostly padding) for 16 KB of weights, and the whole ring of every SM is weights in flight.  Padding rows are neither read nor
// computed nor stored, and the rows of the gate/up projection are picked from x with cp.async, so no dispatch pass runs before it.
// Each sum runs over the same 16-deep steps in the same order as in the pair kernels: same bits.
//
// warp 0 weights (TMA); warp 1 MMA; warps 2, 3, 8 and 9 rows (TMA, or cp.async where they are picked); warps 4-7 epilogue: thread =
// weight column, so the tile goes through shared memory, 32 rows at a time, and leaves row by row.
#pragma once

#include "common.cuh"
#include "grouped_gemm.cuh"
#include "tcgen05.cuh"

namespace lewi {
namespace few {

enum Epi { PLAIN = 0, SWIGLU = 1, LOGITS = 2 };
constexpr int BK = 64;
constexpr int BOX = 64 * 128;                  // bytes of a [64 k][64 columns] box of weights
constexpr int MAX_ROWS = 128;
constexpr int THREADS = 320;
constexpr int LOADERS = 4;                     // warps that bring rows
constexpr int MAX_STAGES = 20;
constexpr int TMEM_COLS = 2 * MAX_ROWS;
constexpr int STAGING_LD = 144;                // floats per row: the 16-byte reads of eight threads (2 rows x 4) meet 32 banks
constexpr int STAGING_BYTES = 32 * STAGING_LD * 4;
constexpr int BAR_BYTES = (2 * MAX_STAGES + 4) * 8 + 16;
constexpr int SMEM_LIMIT = 227 * 1024;
constexpr int RING_LIMIT = SMEM_LIMIT - STAGING_BYTES - BAR_BYTES;
// LOGITS: 64 columns per tile (more CTAs for the few columns there are), two 64-deep steps per stage: 0.27 us a step went to the
// single-threaded loops around them, whatever was loaded or multiplied.
template <int EPI> __host__ __device__ constexpr int steps_per_stage() { return EPI == LOGITS ? 2 : 1; }
template <int EPI> __host__ __device__ constexpr int tile_cols() { return EPI == PLAIN ? 128 : 64; }           // output columns per tile (SWIGLU: 64 of g, 64 of u)

struct Args {
  // several groups: row blocks of 128, expert and rows of each from the routing tables; experts of more than max_group rows are left out
  const int32_t* block_expert;   // null: one group
  const int32_t* n_blocks;
  const int32_t* pad_offsets;
  const int32_t* counts;
  int max_group;
  int E;
  int units;                     // bound on / number of row blocks
  int unit_rows;                 // one group: rows per unit, a multiple of 16
  long long rows;                // one group: rows in all
  // rows picked by index (null: the rows of the block lie at its place): row r is gather_idx[r] / gather_div, zeros where negative
  const int32_t* gather_idx;
  int gather_div;
  const __nv_bfloat16* x;        // [.][K]
  int K;
  int kb_total, k_wrap;          // k_wrap > 0: the rows' k coordinate wraps there
  int N, n_tiles;                // output columns (SWIGLU: f)
  int stages, stage_bytes, row_bytes;   // row_bytes: room for the rows of one 64-deep step
  void* out;                     // PLAIN bf16 [rows,N]; SWIGLU h [rows,f]; LOGITS f32 [rows,N]
  __nv_bfloat16* gu;             // SWIGLU: [rows][2][f] or null
  const int32_t* scale_idx;      // SWIGLU: h of row r is multiplied by scale_src[scale_idx[r]] (null index: by scale_src[r])
  const float* scale_src;
  const float* col_bias;         // LOGITS: f32 [N] or null
  uint64_t desc_hi_w, desc_hi_r;
  uint32_t idesc;                // without N
  // Launched early (common.cuh): only the rows are waited for, since the weights and the routing tables are older than the kernel before
  // this one, which had itself waited for them when it let this one start; otherwise everything is.
  int rows_only;
};

struct Tile {
  int e, row0, valid, rows16, n0;   // rows16: valid rounded up to 16; 0: nothing to do
};

// Barriers of the four epilogue warps.  bar.* wants each warp converged, which is not left to how the compiler joins the lanes of a wait
// that they leave at different turns, or of a branch.
__device__ __forceinline__ void epi_sync() {
  __syncwarp();
  asm volatile("bar.sync 1, 128;" ::: "memory");
}
// the same barrier; whether p holds in one of the threads
__device__ __forceinline__ bool epi_any(bool p) {
  uint32_t r;
  __syncwarp();
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbar.red.or.pred q, 1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(r) : "r"((uint32_t)p) : "memory");
  return r != 0;
}

template <int EPI>
__device__ __forceinline__ Tile decode(const Args& a, int tile, int total) {
  Tile t{0, 0, 0, 0, 0};
  if (tile >= total) return t;
  const int unit = tile / a.n_tiles;
  t.n0 = (tile - unit * a.n_tiles) * tile_cols<EPI>();
  if (a.block_expert != nullptr) {
    t.row0 = unit * MAX_ROWS;
    t.e = a.block_expert[unit];
    if (t.e < 0 || t.e >= a.E) return t;   // corrupted table: every role skips the tile
    const int rows = a.counts[t.e];
    t.valid = rows > a.max_group ? 0 : min(MAX_ROWS, rows - (t.row0 - a.pad_offsets[t.e]));
  } else {
    t.row0 = unit * a.unit_rows;
    t.valid = (int)min((long long)a.unit_rows, a.rows - t.row0);
  }
  t.rows16 = max(0, (t.valid + 15) & ~15);
  return t;
}

template <int EPI>
__global__ void __launch_bounds__(THREADS, 1)
few_gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_w2, const __grid_constant__ CUtensorMap tm_r,
                const Args a) {
  constexpr int W_BYTES = 2 * BOX, KPS = steps_per_stage<EPI>();
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t base = ptx::smem_u32(smem_raw);
  if ((base & 1023u) != 0) {
    if (threadIdx.x == 0) raise_status(LEWI_STATUS_SMEM_LAYOUT);
    return;
  }
  const int ring = a.stages * a.stage_bytes;
  float* staging = reinterpret_cast<float*>(smem_raw + ring);
  const uint32_t bars = base + ring + STAGING_BYTES;
  auto full_bar = [&](int s) { return bars + 8u * s; };
  auto empty_bar = [&](int s) { return bars + 8u * (MAX_STAGES + s); };
  auto tfull_bar = [&](int b) { return bars + 8u * (2 * MAX_STAGES + b); };
  auto tempty_bar = [&](int b) { return bars + 8u * (2 * MAX_STAGES + 2 + b); };
  uint8_t* tail = smem_raw + ring + STAGING_BYTES + (2 * MAX_STAGES + 4) * 8;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(tail);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tail + 8);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    for (int s = 0; s < a.stages; ++s) {
      ptx::mbar_init(full_bar(s), a.gather_idx != nullptr ? 1 + 32 * LOADERS : 1);   // the byte count's arrival, those of the copying lanes
      ptx::mbar_init(empty_bar(s), 1);
    }
    for (int b = 0; b < 2; ++b) {
      ptx::mbar_init(tfull_bar(b), 1);
      ptx::mbar_init(tempty_bar(b), 4);
    }
    *abort_flag = 0;
    ptx::mbar_fence_init();
    ptx::fence_proxy_async();
    ptx::prefetch_tensormap(&tm_w);
    if constexpr (EPI == SWIGLU) ptx::prefetch_tensormap(&tm_w2);
    ptx::prefetch_tensormap(&tm_r);
  }
  if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), TMEM_COLS);
    ptx::tmem_relinquish();
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (!a.rows_only) {
    grid_wait();
    grid_launch();   // (after the wait: what starts now may count on everything before THIS kernel)
  }
  const int n_units = a.n_blocks != nullptr ? min(a.units, max(a.n_blocks[0], 0)) : a.units;
  const int total = n_units * a.n_tiles, step = (int)gridDim.x;

  if (warp == 0) {
    // ------------------------------------------------------------------ weights
    if (ptx::elect_one()) {
      int s = 0;
      uint32_t ph = 0;
      bool ok = true;
      Tile next = decode<EPI>(a, blockIdx.x, total);
      for (int tile = blockIdx.x; ok && tile < total; tile += step) {
        const Tile t = next;
        next = decode<EPI>(a, tile + step, total);
        if (t.rows16 == 0) continue;
        const int row_tx = a.gather_idx != nullptr ? 0 : t.rows16 * 128;
        for (int kb = 0; kb < a.kb_total; kb += KPS) {
          if (!ptx::mbar_wait(empty_bar(s), ph ^ 1u, abort_flag)) { ok = false; break; }
          const uint32_t w = base + s * a.stage_bytes;
          if constexpr (EPI == LOGITS) {
            const bool two = kb + 1 < a.kb_total;
            ptx::mbar_expect_tx(full_bar(s), two ? 2 * (BOX + row_tx) : BOX + row_tx);
            ptx::tma_load_3d(w, &tm_w, full_bar(s), t.n0, kb * BK, 0);
            if (two) ptx::tma_load_3d(w + BOX, &tm_w, full_bar(s), t.n0, kb * BK + BK, 0);
          } else {
            ptx::mbar_expect_tx(full_bar(s), W_BYTES + row_tx);
            ptx::tma_load_3d(w, &tm_w, full_bar(s), t.n0, kb * BK, t.e);
            if constexpr (EPI == SWIGLU) ptx::tma_load_3d(w + BOX, &tm_w2, full_bar(s), t.n0, kb * BK, t.e);
            else ptx::tma_load_3d(w + BOX, &tm_w, full_bar(s), t.n0 + 64, kb * BK, t.e);
          }
          if (++s == a.stages) { s = 0; ph ^= 1u; }
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA
    if (ptx::elect_one()) {
      int s = 0;
      uint32_t ph = 0, acc_it = 0;
      bool ok = true;
      Tile next = decode<EPI>(a, blockIdx.x, total);
      for (int tile = blockIdx.x; ok && tile < total; tile += step) {
        const Tile t = next;
        next = decode<EPI>(a, tile + step, total);
        if (t.rows16 == 0) continue;
        const uint32_t acc = acc_it & 1u;
        if (!ptx::mbar_wait(tempty_bar(acc), ((acc_it >> 1) & 1u) ^ 1u, abort_flag)) break;
        ptx::tc_fence_after();
        const uint32_t idesc = a.idesc | (uint32_t)(t.rows16 >> 3) << 17;
        for (int kb = 0; kb < a.kb_total; kb += KPS) {
          if (!ptx::mbar_wait(full_bar(s), ph, abort_flag)) { ok = false; break; }
          if (a.gather_idx != nullptr) ptx::fence_proxy_async();   // the rows were written through the generic proxy
          ptx::tc_fence_after();
          const uint32_t w = base + s * a.stage_bytes, r = w + W_BYTES;
#pragma unroll
          for (int b = 0; b < KPS; ++b) {
            if (b > 0 && kb + b >= a.kb_total) break;
#pragma unroll
            for (int j = 0; j < BK / 16; ++j)   // (LOGITS: rows 64.. of the M side are whatever follows the box; nobody reads their results)
              ptx::mma_bf16(tmem_base + acc * MAX_ROWS, ptx::smem_desc(a.desc_hi_w, w + b * BOX + j * 2048),
                            ptx::smem_desc(a.desc_hi_r, r + b * a.row_bytes + j * 32), idesc, (kb > 0 || b > 0 || j > 0) ? 1u : 0u);
          }
          ptx::mma_commit(empty_bar(s));
          if (++s == a.stages) { s = 0; ph ^= 1u; }
        }
        if (!ok) break;
        ptx::mma_commit(tfull_bar(acc));
        ++acc_it;
      }
    }
    __syncwarp();
  } else if (warp < 4 || warp >= 8) {
    // ------------------------------------------------------------------ rows
    const int ld = warp < 4 ? warp - 2 : warp - 6;
    const int stages_per_tile = (a.kb_total + KPS - 1) / KPS;
    grid_wait();
    uint32_t it0 = 0;
    Tile next = decode<EPI>(a, blockIdx.x, total);
    for (int tile = blockIdx.x; tile < total; tile += step) {
      const Tile t = next;
      next = decode<EPI>(a, tile + step, total);
      if (t.rows16 == 0) continue;
      int s = (int)(it0 % (uint32_t)a.stages);
      uint32_t ph = (it0 / (uint32_t)a.stages) & 1u;
      bool ok = true;
      if (a.gather_idx != nullptr) {
        // rows 16*i + 4*ld + lane/8 of the tile, 16-byte piece lane % 8 of each
        const int sub = ld * 4 + (lane >> 3), piece = lane & 7;
        const __nv_bfloat16* src[8];
        uint32_t have = 0;   // bit i: the row has a token
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int slot = i * 16 < t.rows16 ? a.gather_idx[t.row0 + i * 16 + sub] : -1;
          src[i] = a.x + (slot < 0 ? 0 : (long long)((unsigned)slot / (unsigned)a.gather_div) * a.K + piece * 8);
          have |= (slot < 0 ? 0u : 1u) << i;
        }
        const uint32_t dst = base + W_BYTES + sub * 128 + ((piece ^ (sub & 7)) << 4);
        for (int k = 0; k < a.kb_total * BK; k += BK) {
          ok = __all_sync(0xffffffffu, ptx::mbar_wait(empty_bar(s), ph ^ 1u, abort_flag));
          if (!ok) break;
          const uint32_t in = k + piece * 8 < a.K ? have : 0u, at = dst + s * a.stage_bytes;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if (i * 16 >= t.rows16) break;
            ptx::cp_async16(at + i * 2048, (in >> i & 1u) ? src[i] + k : a.x, (in >> i & 1u) * 16u);
          }
          ptx::cp_async_arrive(full_bar(s));
          if (++s == a.stages) { s = 0; ph ^= 1u; }
        }
      } else if (ld < KPS && ptx::elect_one()) {   // a loader per 64-deep step of the stage
        int k = ld * BK;
        for (int kb = ld; kb < a.kb_total; kb += KPS) {
          if (!ptx::mbar_wait(empty_bar(s), ph ^ 1u, abort_flag)) { ok = false; break; }
          while (a.k_wrap > 0 && k >= a.k_wrap) k -= a.k_wrap;
          const uint32_t r = base + s * a.stage_bytes + W_BYTES + ld * a.row_bytes;
          for (int x = 0; x < t.rows16; x += 16) ptx::tma_load_2d(r + x * 128, &tm_r, full_bar(s), k, t.row0 + x);
          k += KPS * BK;
          if (++s == a.stages) { s = 0; ph ^= 1u; }
        }
      }
      it0 += stages_per_tile;
      if (!__all_sync(0xffffffffu, ok)) break;
    }
    ptx::cp_async_wait_all();
  } else {
    // ------------------------------------------------------------------ epilogue
    const int tid = threadIdx.x - 128, grp = warp & 3;
    grid_wait();
    uint32_t acc_it = 0;
    Tile next = decode<EPI>(a, blockIdx.x, total);
    for (int tile = blockIdx.x; tile < total; tile += step) {
      const Tile t = next;
      next = decode<EPI>(a, tile + step, total);
      if (t.rows16 == 0) continue;
      const uint32_t acc = acc_it & 1u;
      // the four warps go on or leave together: one that left alone would keep the others at the barriers below
      const bool got = ptx::mbar_wait(tfull_bar(acc), (acc_it >> 1) & 1u, abort_flag);
      if (epi_any(!got)) break;
      ptx::tc_fence_after();
      for (int c = 0; c < t.rows16; c += 32) {
        uint32_t v[32];
        ptx::tmem_ld_32x32(tmem_base + acc * MAX_ROWS + c + ((uint32_t)(grp * 32) << 16), v);
        ptx::tmem_ld_wait();
        if (c + 32 >= t.rows16) {
          ptx::tc_fence_before();
          __syncwarp();
          if (lane == 0) ptx::mbar_arrive(tempty_bar(acc));
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) staging[j * STAGING_LD + grp * 32 + lane] = __uint_as_float(v[j]);
        epi_sync();
        const int r = tid >> 2, q = tid & 3;
        const long long row = (long long)t.row0 + c + r;
        if (c + r < t.valid) {
          const float* src = staging + r * STAGING_LD + q * 4;
          if constexpr (EPI == SWIGLU) {
            float sc = 1.f;
            if (a.scale_src != nullptr) {
              const long long gi = a.scale_idx != nullptr ? (long long)a.scale_idx[row] : row;
              sc = gi >= 0 ? a.scale_src[gi] : 0.f;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int n = t.n0 + i * 16 + q * 4;
              if (n >= a.N) break;
              const float4 g = *reinterpret_cast<const float4*>(src + i * 16), u = *reinterpret_cast<const float4*>(src + 64 + i * 16);
              auto act = [&](float x, float y) { return x * gg::fast_sigmoid(x) * y * sc; };
              *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(a.out) + row * a.N + n) =
                  make_uint2(pack_bf16(act(g.x, u.x), act(g.y, u.y)), pack_bf16(act(g.z, u.z), act(g.w, u.w)));
              if (a.gu != nullptr) {
                *reinterpret_cast<uint2*>(a.gu + row * 2 * a.N + n) = make_uint2(pack_bf16(g.x, g.y), pack_bf16(g.z, g.w));
                *reinterpret_cast<uint2*>(a.gu + (row * 2 + 1) * a.N + n) = make_uint2(pack_bf16(u.x, u.y), pack_bf16(u.z, u.w));
              }
            }
          } else if constexpr (EPI == PLAIN) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const int n = t.n0 + i * 16 + q * 4;
              if (n >= a.N) break;
              const float4 x = *reinterpret_cast<const float4*>(src + i * 16);
              *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(a.out) + row * a.N + n) =
                  make_uint2(pack_bf16(x.x, x.y), pack_bf16(x.z, x.w));
            }
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int n = t.n0 + i * 16 + q * 4;
              if (n >= a.N) break;
              float4 x = *reinterpret_cast<const float4*>(src + i * 16);
              if (a.col_bias != nullptr) { x.x += a.col_bias[n]; x.y += a.col_bias[n + 1]; x.z += a.col_bias[n + 2]; x.w += a.col_bias[n + 3]; }
              *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.out) + row * a.N + n) = x;
            }
          }
        }
        epi_sync();
      }
      if constexpr (EPI == SWIGLU) {
        // the block's padding rows of h: zeros, so that a weight gradient may contract over whole blocks
        if (a.block_expert != nullptr) {
          for (int r = t.valid + (tid >> 3); r < MAX_ROWS; r += 16) {
            const int n = t.n0 + (tid & 7) * 8;
            if (n < a.N) st_v4(reinterpret_cast<__nv_bfloat16*>(a.out) + ((long long)t.row0 + r) * a.N + n, make_uint4(0, 0, 0, 0));
          }
        }
      }
      ++acc_it;
    }
  }

  ptx::tc_fence_before();
  __syncthreads();
  if (*abort_flag) {   // copies and MMAs in flight get a bounded time before shared memory and TMEM go
    const unsigned long long t0 = ptx::globaltimer_ns();
    while (ptx::globaltimer_ns() - t0 < 4000000ull) {
    }
    __syncthreads();
  }
  if (warp == 1) {
    __syncwarp();
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem_base, TMEM_COLS);
  }
}

template <int EPI>
inline int launch(cudaStream_t st, const CUtensorMap& tw, const CUtensorMap& tw2, const CUtensorMap& tr, Args a, int max_rows, bool early = false) {
  static bool attr_set[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return LEWI_ERR_CUDA;
  auto kern = few_gemm_kernel<EPI>;
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT) != cudaSuccess) {
      (void)cudaGetLastError();
      return LEWI_ERR_CUDA;
    }
    attr_set[dev] = true;
  }
  const gg::DescGeometry g;
  a.desc_hi_w = ptx::smem_desc_hi_sw128(g.mn_lbo, g.mn_sbo);
  a.desc_hi_r = ptx::smem_desc_hi_sw128(g.k_lbo, g.k_sbo);
  a.idesc = ptx::instr_desc_bf16(128, 0, 1, 0);
  a.n_tiles = (a.N + tile_cols<EPI>() - 1) / tile_cols<EPI>();
  const int rows16 = max_rows >= MAX_ROWS ? MAX_ROWS : (max_rows + 15) / 16 * 16;
  a.row_bytes = rows16 * 128;   // (a multiple of 1024: tiles start on 1024 bytes)
  a.stage_bytes = 2 * BOX + steps_per_stage<EPI>() * a.row_bytes;
  a.stages = RING_LIMIT / a.stage_bytes;
  if (a.stages > MAX_STAGES) a.stages = MAX_STAGES;
  const long long tiles = (long long)a.units * a.n_tiles;
  if (tiles <= 0) return LEWI_OK;
  if (tiles > 0x7fffffffLL) return LEWI_ERR_LIMIT;
  long long grid = num_sms();
  if (gg::cta_limit() > 0 && grid > gg::cta_limit()) grid = gg::cta_limit();
  if (grid > tiles) grid = tiles;
  const int smem = a.stages * a.stage_bytes + STAGING_BYTES + BAR_BYTES;
  (void)launch_kernel(kern, (int)grid, THREADS, (size_t)smem, st, early, tw, tw2, tr, a);
  LEWI_CHECK_LAUNCH();
  return LEWI_OK;
}

}  // namespace few
}  // namespace lewi
