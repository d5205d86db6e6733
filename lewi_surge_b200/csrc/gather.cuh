// Row-gather kernels: the only data movement of dispatch / combine and of their gradients.
// One warp owns one output row; every lane moves 16-byte pieces, so a 2 KB bf16 row is four
// independent 128-bit loads per lane and the whole warp's traffic is fully coalesced.
// Semantics follow gather_rows / gather_reduce / gather_dot of the reference
// (modal/moe_permute.py:116-158, 161-225, 228-234): multiply and accumulate in float32.
#pragma once

#include "common.cuh"

namespace lewi {

constexpr int kGatherThreads = 256;

template <typename T>
struct Elem;  // 16-byte vector <-> 4 or 8 floats

template <>
struct Elem<float> {
  static constexpr int kPerVec = 4;
  __device__ static __forceinline__ void unpack(uint4 v, float* f) {
    f[0] = __uint_as_float(v.x); f[1] = __uint_as_float(v.y);
    f[2] = __uint_as_float(v.z); f[3] = __uint_as_float(v.w);
  }
  __device__ static __forceinline__ uint4 pack(const float* f) {
    return make_uint4(__float_as_uint(f[0]), __float_as_uint(f[1]), __float_as_uint(f[2]), __float_as_uint(f[3]));
  }
};

template <>
struct Elem<__nv_bfloat16> {
  static constexpr int kPerVec = 8;
  __device__ static __forceinline__ void unpack(uint4 v, float* f) {
    f[0] = bf16_lo(v.x); f[1] = bf16_hi(v.x); f[2] = bf16_lo(v.y); f[3] = bf16_hi(v.y);
    f[4] = bf16_lo(v.z); f[5] = bf16_hi(v.z); f[6] = bf16_lo(v.w); f[7] = bf16_hi(v.w);
  }
  __device__ static __forceinline__ uint4 pack(const float* f) {
    return make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
  }
};

// out[i] = x[src(i)] * scale.  VPL = 16-byte vectors per lane (row bytes <= VPL*512).
template <typename T, int VPL>
__global__ void __launch_bounds__(kGatherThreads) gather_rows_kernel(
    const T* __restrict__ x, const int32_t* __restrict__ idx, const float* __restrict__ scale, T* __restrict__ out,
    long long n_src, long long m, int d, int idx_div, int scale_by_idx, const int32_t* __restrict__ n_rows_dev,
    int rows_per_unit) {
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  long long rows = m;
  if (n_rows_dev != nullptr) rows = min(rows, (long long)n_rows_dev[0] * rows_per_unit);
  const int nvec = d / Elem<T>::kPerVec;
  for (long long i = warp0; i < rows; i += n_warps) {
    const int raw = idx[i];
    long long src = raw;
    if (idx_div > 1 && raw >= 0) src = raw / idx_div;
    const bool zero = raw < 0;
    if (!zero && src >= n_src) {
      if (lane == 0) raise_status(LEWI_STATUS_BAD_INDEX);
      continue;
    }
    uint4 v[VPL];
#pragma unroll
    for (int c = 0; c < VPL; ++c) {
      int vi = lane + c * kWarp;
      v[c] = make_uint4(0, 0, 0, 0);
      if (!zero && vi < nvec) v[c] = ld_nc_v4(reinterpret_cast<const uint4*>(x + src * d) + vi);
    }
    if (scale != nullptr && !zero) {
      const float s = scale[scale_by_idx ? (long long)raw : i];
#pragma unroll
      for (int c = 0; c < VPL; ++c) {
        float f[Elem<T>::kPerVec];
        Elem<T>::unpack(v[c], f);
#pragma unroll
        for (int q = 0; q < Elem<T>::kPerVec; ++q) f[q] *= s;
        v[c] = Elem<T>::pack(f);
      }
    }
#pragma unroll
    for (int c = 0; c < VPL; ++c) {
      int vi = lane + c * kWarp;
      if (vi < nvec) st_v4(reinterpret_cast<uint4*>(out + i * d) + vi, v[c]);
    }
  }
}

// Dispatch in token order: out[pos[t,j]] = x[t] for the k slots of token t; padded rows that hold no slot
// (row_slot[r] < 0) become zero rows.  Every output row has exactly one writer, so this is the same function as
// the row gather out[r] = x[row_slot[r] / k] -- but each source row is read once instead of k times at k distant
// moments, which keeps the read side at T rows of DRAM traffic however large the source is against the L2.
// A warp looks at ZR rows at a time for those to zero: 4 while no warp of the grid looks more than twice (kZeroRows), since at decode
// sizes nearly all rows are such rows (8 tokens over 128 experts: 6.1 MB of zeros; 13 us with 32 rows per warp, 7 us with 4);
// 32 beyond, where hardly any are (k = 6, d = 256: 16,384 tokens over 16 experts 9.3 us with 4 and 9.8 with 32, 49,152 34 and 32,
// 65,536 over 128 48 and 45).
constexpr int kZeroRows = 4;
template <int VPL, int ZR>
__global__ void __launch_bounds__(kGatherThreads) dispatch_rows_kernel(
    const __nv_bfloat16* __restrict__ x, const int32_t* __restrict__ pos, const int32_t* __restrict__ row_slot,
    __nv_bfloat16* __restrict__ out, long long n_tokens, int k, int d, long long out_rows,
    const int32_t* __restrict__ n_rows_dev, int rows_per_unit) {
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  const int nvec = d / 8;
  long long rows = out_rows;
  if (n_rows_dev != nullptr) rows = min(rows, (long long)n_rows_dev[0] * rows_per_unit);
  for (long long t = warp0; t < n_tokens; t += n_warps) {
    const int my_pos = lane < k ? pos[t * k + lane] : -1;
    uint4 v[VPL];
#pragma unroll
    for (int c = 0; c < VPL; ++c) {
      const int vi = lane + c * kWarp;
      v[c] = make_uint4(0, 0, 0, 0);
      if (vi < nvec) v[c] = ld_nc_v4(reinterpret_cast<const uint4*>(x + t * d) + vi);
    }
    for (int j = 0; j < k; ++j) {
      const long long p = __shfl_sync(0xffffffffu, my_pos, j);
      if (p < 0 || p >= rows) {
        if (lane == 0 && p >= rows) raise_status(LEWI_STATUS_BAD_INDEX);
        continue;
      }
#pragma unroll
      for (int c = 0; c < VPL; ++c) {
        const int vi = lane + c * kWarp;
        if (vi < nvec) st_v4(reinterpret_cast<uint4*>(out + p * d) + vi, v[c]);
      }
    }
  }
  // zero rows of the padded layout
  for (long long r0 = warp0 * ZR; r0 < rows; r0 += n_warps * ZR) {
    const long long r = r0 + lane;
    const unsigned empty = __ballot_sync(0xffffffffu, lane < ZR && r < rows && row_slot[r] < 0);
    for (unsigned m = empty; m != 0; m &= m - 1) {
      const long long rr = r0 + (__ffs(m) - 1);
      for (int vi = lane; vi < nvec; vi += kWarp) st_v4(reinterpret_cast<uint4*>(out + rr * d) + vi, make_uint4(0, 0, 0, 0));
    }
  }
}

// Rows of the unpadded operators, table by table: row r of the sorted order belongs to slot order[r] (negative: to none), slot s sits at row
// pos[s] (negative: nowhere).  The kernels below go through the tokens in order and write the rows that their slots sit at; the two tables
// need not be inverse permutations of one another (a caller may drop slots), so a slot writes the row only if the row names it back, and
// the rows left over, which no slot writes, are visited apart: each row is written once, with what `order` says of it.
__device__ __forceinline__ int slot_of_row(const int32_t* __restrict__ order, long long r, long long n_rows) { return r < n_rows ? order[r] : -1; }
// Which of a warp's 32 rows are left over, lane's row being r of slot s; the slots write rows below n_slot_rows.
__device__ __forceinline__ unsigned left_over(const int32_t* __restrict__ pos, int s, long long r, long long n_rows, long long n_slot_rows,
                                              long long n_slots) {
  if (s >= n_slots) raise_status(LEWI_STATUS_BAD_INDEX);
  return __ballot_sync(0xffffffffu, r < n_rows && s < n_slots && (s < 0 || r >= n_slot_rows || pos[s] != r));
}
// put(row, slot) writes row `row` for slot `slot` (negative: zeros); whole warp.
template <class Put>
__device__ __forceinline__ void put_left_over(unsigned left, long long r0, int s, Put put) {
  for (; left != 0; left &= left - 1) {
    const int from = __ffs(left) - 1;
    put(r0 + from, __shfl_sync(0xffffffffu, s, from));
  }
}
// The row of this lane's slot, -1 where nothing is to be written for it.  Without `order` pos is a permutation: a slot without a row is an error.
__device__ __forceinline__ int row_of_slot(const int32_t* __restrict__ order, int p, long long slot, long long n_rows) {
  const bool in = p >= 0 && p < n_rows;
  if (order == nullptr && !in) raise_status(LEWI_STATUS_BAD_INDEX);
  return in && (order == nullptr || order[p] == slot) ? p : -1;
}

// out[r] = x[order[r] / k], in token order: every row of x is read once.  Between events, this | the row gather, in us: 16,384 tokens, k = 12,
// d = 2048, bf16 152 | 248; 5000 tokens, k = 6, d = 1024, float32 31 | 39.  (Looking for rows left over after the tokens: 155 and 35.)
// A warp writes the k rows of its token one after the other, so with few tokens the gather, a warp per row, is the faster one: d = 2048,
// bf16, k = 12: 60 tokens 12 | 8, 1200 20.5 | 18.4, 2400 28.7 | 34.8; d = 1024, float32, k = 6: 60 tokens 10 | 8, 1200 14.4 | 14.2, 2400
// 18.5 | 20.5.  The line lies at kDispatchWarps tokens per SM.
constexpr int kDispatchWarps = 10;
template <typename T, int VPL>
__global__ void __launch_bounds__(kGatherThreads) dispatch_tokens_kernel(const T* __restrict__ x, const int32_t* __restrict__ order,
                                                                         const int32_t* __restrict__ pos, T* __restrict__ out,
                                                                         long long n_tokens, int k, int d) {
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5, rows = n_tokens * k;
  const int nvec = d / Elem<T>::kPerVec;
  auto put = [&](long long r, int s) {
    const uint4* src = reinterpret_cast<const uint4*>(x + (long long)(s < 0 ? 0 : s / k) * d);
#pragma unroll 1
    for (int vi = lane; vi < nvec; vi += kWarp) st_v4(reinterpret_cast<uint4*>(out + r * d) + vi, s < 0 ? make_uint4(0, 0, 0, 0) : ld_nc_v4(src + vi));
  };
  // (k <= 32: there are no more looks of 32 rows than tokens, so a warp has one beside each of its tokens and the loads of both in flight)
  for (long long t = warp0; t < n_tokens; t += n_warps) {
    const int my_pos = lane < k ? pos[t * k + lane] : -1, look = order != nullptr ? slot_of_row(order, t * kWarp + lane, rows) : -1;
    uint4 v[VPL];
#pragma unroll
    for (int c = 0; c < VPL; ++c) {
      const int vi = lane + c * kWarp;
      v[c] = make_uint4(0, 0, 0, 0);
      if (vi < nvec) v[c] = ld_nc_v4(reinterpret_cast<const uint4*>(x + t * d) + vi);
    }
    const int my_row = lane < k ? row_of_slot(order, my_pos, t * k + lane, rows) : -1;
    const unsigned left = order != nullptr ? left_over(pos, look, t * kWarp + lane, rows, rows, rows) : 0u;
    for (int j = 0; j < k; ++j) {
      const long long p = __shfl_sync(0xffffffffu, my_row, j);
      if (p < 0) continue;
#pragma unroll
      for (int c = 0; c < VPL; ++c) {
        const int vi = lane + c * kWarp;
        if (vi < nvec) st_v4(reinterpret_cast<uint4*>(out + p * d) + vi, v[c]);
      }
    }
    put_left_over(left, t * kWarp, look, put);
  }
}

// out[t] = sum_j w[t,j] * y[pos[t,j]] (+ add0[t] + add1[t]); f32 accumulate.
template <typename TI, typename TO, int VPL>
__global__ void __launch_bounds__(kGatherThreads) gather_reduce_kernel(
    const TI* __restrict__ y, const int32_t* __restrict__ pos, const float* __restrict__ w,
    const TI* __restrict__ add0, const TI* __restrict__ add1, TO* __restrict__ out, long long n, int k, int d,
    long long n_y_rows) {
  constexpr int PV = Elem<TI>::kPerVec;
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  const int nvec = d / PV;
  for (long long t = warp0; t < n; t += n_warps) {
    float acc[VPL][PV];
#pragma unroll
    for (int c = 0; c < VPL; ++c)
#pragma unroll
      for (int q = 0; q < PV; ++q) acc[c][q] = 0.f;
    int my_pos = 0;
    float my_w = 1.f;
    if (lane < k) {
      my_pos = pos[t * k + lane];
      if (w != nullptr) my_w = w[t * k + lane];
    }
    for (int j = 0; j < k; ++j) {
      const long long p = __shfl_sync(0xffffffffu, my_pos, j);
      const float wj = __shfl_sync(0xffffffffu, my_w, j);
      if (p < 0 || p >= n_y_rows) {
        if (lane == 0 && p >= n_y_rows) raise_status(LEWI_STATUS_BAD_INDEX);
        continue;
      }
      uint4 v[VPL];
#pragma unroll
      for (int c = 0; c < VPL; ++c) {
        int vi = lane + c * kWarp;
        v[c] = make_uint4(0, 0, 0, 0);
        if (vi < nvec) v[c] = ld_nc_v4(reinterpret_cast<const uint4*>(y + p * d) + vi);
      }
#pragma unroll
      for (int c = 0; c < VPL; ++c) {
        float f[PV];
        Elem<TI>::unpack(v[c], f);
#pragma unroll
        for (int q = 0; q < PV; ++q) acc[c][q] = fmaf(wj, f[q], acc[c][q]);
      }
    }
#pragma unroll
    for (int a = 0; a < 2; ++a) {
      const TI* add = a == 0 ? add0 : add1;
      if (add == nullptr) continue;
#pragma unroll
      for (int c = 0; c < VPL; ++c) {
        int vi = lane + c * kWarp;
        if (vi < nvec) {
          float f[PV];
          Elem<TI>::unpack(ld_nc_v4(reinterpret_cast<const uint4*>(add + t * d) + vi), f);
#pragma unroll
          for (int q = 0; q < PV; ++q) acc[c][q] += f[q];
        }
      }
    }
    // store: PV input elements per vector -> PV output elements
#pragma unroll
    for (int c = 0; c < VPL; ++c) {
      int vi = lane + c * kWarp;
      if (vi >= nvec) continue;
      TO* o = out + t * d + (long long)vi * PV;
      if constexpr (sizeof(TO) == 4) {
#pragma unroll
        for (int q = 0; q < PV; q += 4) st_v4(reinterpret_cast<float*>(o) + q, Elem<float>::pack(&acc[c][q]));
      } else {
        if constexpr (PV == 8) {
          st_v4(o, Elem<__nv_bfloat16>::pack(acc[c]));
        } else {
          uint2 pk = make_uint2(pack_bf16(acc[c][0], acc[c][1]), pack_bf16(acc[c][2], acc[c][3]));
          *reinterpret_cast<uint2*>(o) = pk;
        }
      }
    }
  }
}

// The same for few rows, same bits: a warp takes 32 vectors of one row of `out` and has eight rows of y in flight.  The kernel
// above walks the k rows of a token one trip to memory after the other, which is what a small call takes
// (8 tokens, k = 6, d = 1024: 10.2 us, here 4.1; 64 tokens, k = 8, d = 2048: 23 and 5.1 us; 1000 tokens, k = 6: 10.7 and 6.1).
// It reads positions and weights once per 32 vectors, so where the trips are few (small k) or short rows give the row kernel warps
// enough, that one is quicker from some size on.  Measured line between them (k 1 to 12, d 128 to 4096, bf16 and float32, 300 to
// 9500 warps, sources in L2): gather_reduce_few() picks the quicker one within 1 % on average and never one more than 5 % slower.
// Either side of it, in us, this kernel first: bf16 d = 1024, k = 1: 592 rows 2.4 and 2.3, 2368 rows 5.2 and 2.7; k = 6: 1184 rows
// 4.0 and 4.6, 2368 rows 6.5 and 5.2; d = 2048, k = 8: 1184 rows 7.0 and 8.6.
template <typename TI, typename TO>
__global__ void __launch_bounds__(kGatherThreads) gather_reduce_few_kernel(
    const TI* __restrict__ y, const int32_t* __restrict__ pos, const float* __restrict__ w,
    const TI* __restrict__ add0, const TI* __restrict__ add1, TO* __restrict__ out, long long n, int k, int d, int pieces,
    long long n_y_rows) {
  constexpr int PV = Elem<TI>::kPerVec, NJ = 8;
  const int lane = threadIdx.x & 31;
  const long long unit = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long t = unit / pieces;
  if (t >= n) return;
  const int piece = (int)(unit - t * pieces), vi = piece * kWarp + lane;
  const bool live = vi < d / PV;
  int my_pos = 0;
  float my_w = 1.f;
  if (lane < k) {
    my_pos = pos[t * k + lane];
    if (w != nullptr) my_w = w[t * k + lane];
  }
  const uint4 zero = make_uint4(0, 0, 0, 0);
  uint4 va[2] = {zero, zero};
  if (live && add0 != nullptr) va[0] = ld_nc_v4(reinterpret_cast<const uint4*>(add0 + t * d) + vi);
  if (live && add1 != nullptr) va[1] = ld_nc_v4(reinterpret_cast<const uint4*>(add1 + t * d) + vi);
  float acc[PV];
#pragma unroll
  for (int q = 0; q < PV; ++q) acc[q] = 0.f;
  for (int j0 = 0; j0 < k; j0 += NJ) {
    uint4 v[NJ];
#pragma unroll
    for (int x = 0; x < NJ; ++x) {
      const long long p = __shfl_sync(0xffffffffu, my_pos, (j0 + x) & (kWarp - 1));
      v[x] = live && j0 + x < k && p >= 0 && p < n_y_rows ? ld_nc_v4(reinterpret_cast<const uint4*>(y + p * d) + vi) : zero;
    }
#pragma unroll
    for (int x = 0; x < NJ; ++x) {
      const long long p = __shfl_sync(0xffffffffu, my_pos, (j0 + x) & (kWarp - 1));
      const float wj = __shfl_sync(0xffffffffu, my_w, (j0 + x) & (kWarp - 1));
      if (j0 + x >= k) continue;
      if (p < 0 || p >= n_y_rows) {
        if (lane == 0 && piece == 0 && p >= n_y_rows) raise_status(LEWI_STATUS_BAD_INDEX);
        continue;
      }
      float f[PV];
      Elem<TI>::unpack(v[x], f);
#pragma unroll
      for (int q = 0; q < PV; ++q) acc[q] = fmaf(wj, f[q], acc[q]);
    }
  }
#pragma unroll
  for (int a = 0; a < 2; ++a) {
    if ((a == 0 ? add0 : add1) == nullptr) continue;
    float f[PV];
    Elem<TI>::unpack(va[a], f);
#pragma unroll
    for (int q = 0; q < PV; ++q) acc[q] += f[q];
  }
  if (!live) return;
  TO* o = out + t * d + (long long)vi * PV;
  if constexpr (sizeof(TO) == 4) {
#pragma unroll
    for (int q = 0; q < PV; q += 4) st_v4(reinterpret_cast<float*>(o) + q, Elem<float>::pack(&acc[q]));
  } else if constexpr (PV == 8) {
    st_v4(o, Elem<__nv_bfloat16>::pack(acc));
  } else {
    *reinterpret_cast<uint2*>(o) = make_uint2(pack_bf16(acc[0], acc[1]), pack_bf16(acc[2], acc[3]));
  }
}

// Whether a call of `warps` warps goes to the kernel above (see there): more trips (k) and longer rows (d) move the line up.
inline bool gather_reduce_few(long long warps, int k, int d) {
  const int ke = k < 7 ? k : 7;   // (from eight source rows on, in flight at once, more of them do not help)
  const long long line = 4ll * num_sms() * (ke - 1) + (long long)d * (ke + 1) / 2, most = 64ll * num_sms();
  return warps <= (line < most ? line : most);
}

// out[t,j] = <g[t], y[pos[t,j]]>.
template <typename T, int VPL>
__global__ void __launch_bounds__(kGatherThreads) gather_dot_kernel(
    const T* __restrict__ y, const int32_t* __restrict__ pos, const T* __restrict__ g, float* __restrict__ out,
    long long n, int k, int d, long long n_y_rows) {
  constexpr int PV = Elem<T>::kPerVec;
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  const int nvec = d / PV;
  for (long long t = warp0; t < n; t += n_warps) {
    float gv[VPL][PV];
#pragma unroll
    for (int c = 0; c < VPL; ++c) {
      int vi = lane + c * kWarp;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (vi < nvec) v = ld_nc_v4(reinterpret_cast<const uint4*>(g + t * d) + vi);
      Elem<T>::unpack(v, gv[c]);
    }
    int my_pos = (lane < k) ? pos[t * k + lane] : 0;
    float my_out = 0.f;
    for (int j = 0; j < k; ++j) {
      const long long p = __shfl_sync(0xffffffffu, my_pos, j);
      float s = 0.f;
      if (p >= 0 && p < n_y_rows) {
#pragma unroll
        for (int c = 0; c < VPL; ++c) {
          int vi = lane + c * kWarp;
          if (vi < nvec) {
            float f[PV];
            Elem<T>::unpack(ld_nc_v4(reinterpret_cast<const uint4*>(y + p * d) + vi), f);
#pragma unroll
            for (int q = 0; q < PV; ++q) s = fmaf(gv[c][q], f[q], s);
          }
        }
      } else if (lane == 0 && p >= n_y_rows) {
        raise_status(LEWI_STATUS_BAD_INDEX);
      }
      s = warp_sum(s);
      if (lane == j) my_out = s;
    }
    if (lane < k) out[t * k + lane] = my_out;
  }
}

inline int gather_grid(long long rows) {
  const long long warps_per_cta = kGatherThreads / kWarp;
  long long ctas = (rows + warps_per_cta - 1) / warps_per_cta;
  const long long cap = (long long)num_sms() * 16;  // 8 resident CTAs per SM x 2 waves
  if (ctas > cap) ctas = cap;
  if (ctas < 1) ctas = 1;
  return (int)ctas;
}

// Gradients of the combine, both in one pass over y, in token order: dy[r] = w[order[r]] * g[order[r] / k] and dw[t,j] = <g[t], y[pos[t,j]]>,
// g in y's type (a float32 g is rounded here).  Where the tables are inverse permutations a row of g is read once, not k times; a warp
// requests the next row of y while it works on one.
// 5003 tokens, k = 6, d = 1024, float32: 47 us (scaled gather and dots 35 + 39); 16,384 tokens, k = 12, d = 2048, bf16: 328 us, 5.3 TB/s
// (240 + 207 and 32 for the rounded copy of g).  A warp per row of y instead, g out of L2 k times: 55 and 472 us.
// Rows of 8 KB (three of them in a lane's registers, up to 255 and one CTA per SM), between events, this | what it replaces: float32,
// d = 2048, 60 tokens, k = 6 18 | 32, 5003 96 | 148, 16,384, k = 12 539 | 810; bf16, d = 4096, 8000 tokens, k = 12 309 | 513.
template <typename T, typename TG, int VPL>
__global__ void __launch_bounds__(kGatherThreads) combine_bwd_kernel(const T* __restrict__ y, const int32_t* __restrict__ order,
                                                                     const int32_t* __restrict__ pos, const TG* __restrict__ g,
                                                                     const float* __restrict__ w, T* __restrict__ dy, float* __restrict__ dw,
                                                                     long long n, int k, int d, long long n_y_rows, long long n_dy_rows) {
  constexpr int PV = Elem<T>::kPerVec, GV = PV * sizeof(TG) / 16;   // vectors of g per vector of y
  const int lane = threadIdx.x & 31;
  const long long warp0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  const int nvec = d / PV;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  const long long n_rows = min(n_y_rows, n_dy_rows);   // of these the slots take care
  auto g_vec = [&](long long t, int vi) {   // a vector of g[t] in y's type
    if constexpr (GV == 2) {   // float32 -> bf16
      const uint4* src = reinterpret_cast<const uint4*>(g + t * d) + (long long)vi * 2;
      const uint4 a = ld_nc_v4(src), b = ld_nc_v4(src + 1);
      auto two = [](uint32_t lo, uint32_t hi) { return pack_bf16(__uint_as_float(lo), __uint_as_float(hi)); };
      return make_uint4(two(a.x, a.y), two(a.z, a.w), two(b.x, b.y), two(b.z, b.w));
    } else {
      return ld_nc_v4(reinterpret_cast<const uint4*>(g + t * d) + vi);
    }
  };
  for (long long t = warp0; t < n; t += n_warps) {
    const int my_pos = lane < k ? pos[t * k + lane] : -1;
    const int my_row = lane < k ? row_of_slot(order, my_pos, t * k + lane, n_rows) : -1;
    if (my_pos >= n_y_rows) raise_status(LEWI_STATUS_BAD_INDEX);
    const float my_w = lane < k ? w[t * k + lane] : 0.f;
    uint4 gv[VPL], yv[VPL], next[VPL];
    auto fetch = [&](int j, uint4 (&v)[VPL]) {
      const long long p = __shfl_sync(0xffffffffu, my_row, j);
#pragma unroll
      for (int c = 0; c < VPL; ++c) {
        const int vi = lane + c * kWarp;
        v[c] = vi < nvec && p >= 0 ? ld_nc_v4(reinterpret_cast<const uint4*>(y + p * d) + vi) : zero;
      }
    };
    fetch(0, yv);
#pragma unroll
    for (int c = 0; c < VPL; ++c) {
      const int vi = lane + c * kWarp;
      gv[c] = vi < nvec ? g_vec(t, vi) : zero;
    }
    float my_dot = 0.f;
    for (int j = 0; j < k; ++j) {
      if (j + 1 < k) fetch(j + 1, next);
      const long long p = __shfl_sync(0xffffffffu, my_row, j);
      const float s = __shfl_sync(0xffffffffu, my_w, j);
      float dot = 0.f;
#pragma unroll
      for (int c = 0; c < VPL; ++c) {
        const int vi = lane + c * kWarp;
        if (vi < nvec && p >= 0) {
          float f[PV], q[PV];
          Elem<T>::unpack(yv[c], f);
          Elem<T>::unpack(gv[c], q);
#pragma unroll
          for (int e = 0; e < PV; ++e) {
            dot = fmaf(q[e], f[e], dot);
            q[e] *= s;
          }
          st_v4(reinterpret_cast<uint4*>(dy + p * d) + vi, Elem<T>::pack(q));
        }
        yv[c] = next[c];
      }
      dot = warp_sum(dot);
      if (lane == j) my_dot = dot;
    }
    // slots at a row that is another slot's: only their dots
    for (unsigned m = __ballot_sync(0xffffffffu, my_row < 0 && my_pos >= 0 && my_pos < n_y_rows); m != 0; m &= m - 1) {
      const int j = __ffs(m) - 1;
      const long long p = __shfl_sync(0xffffffffu, my_pos, j);
      float dot = 0.f;
#pragma unroll 1
      for (int vi = lane; vi < nvec; vi += kWarp) {
        float f[PV], q[PV];
        Elem<T>::unpack(ld_nc_v4(reinterpret_cast<const uint4*>(y + p * d) + vi), f);
        Elem<T>::unpack(g_vec(t, vi), q);
#pragma unroll
        for (int e = 0; e < PV; ++e) dot = fmaf(q[e], f[e], dot);
      }
      dot = warp_sum(dot);
      if (lane == j) my_dot = dot;
    }
    if (lane < k) dw[t * k + lane] = my_dot;
  }
  if (order == nullptr) return;
  auto put = [&](long long r, int s) {
    const float sc = s < 0 ? 0.f : w[s];
#pragma unroll 1
    for (int vi = lane; vi < nvec; vi += kWarp) {
      uint4 v = zero;
      if (s >= 0) {
        float q[PV];
        Elem<T>::unpack(g_vec(s / k, vi), q);
#pragma unroll
        for (int e = 0; e < PV; ++e) q[e] *= sc;
        v = Elem<T>::pack(q);
      }
      st_v4(reinterpret_cast<uint4*>(dy + r * d) + vi, v);
    }
  };
  for (long long r0 = warp0 * kWarp; r0 < n_dy_rows; r0 += n_warps * kWarp) {
    const int look = slot_of_row(order, r0 + lane, n_dy_rows);
    put_left_over(left_over(pos, look, r0 + lane, n_dy_rows, n_rows, n * k), r0, look, put);
  }
}

// Padded rows of the experts that have more than one row block: row r = x[row_slot[r] / k], zeros where row_slot[r] < 0; other experts'
// blocks are passed over.  A CTA takes 16 rows, two per warp (a block per CTA, 16 rows per warp: 15 us instead of 4 for eight experts of
// 700 rows, and the experts' GEMMs wait for it).
constexpr int kHeavyRows = 16;
__global__ void __launch_bounds__(256) gather_heavy_kernel(const __nv_bfloat16* __restrict__ x, const int32_t* __restrict__ row_slot,
                                                           const int32_t* __restrict__ block_expert, const int32_t* __restrict__ n_blocks,
                                                           const int32_t* __restrict__ counts, __nv_bfloat16* __restrict__ out, int max_blocks,
                                                           int k, int d) {
  constexpr int kBlockRows = 128, kParts = kBlockRows / kHeavyRows;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, units = min(max_blocks, n_blocks[0]) * kParts;
  for (int u = blockIdx.x; u < units; u += gridDim.x) {
    if (counts[block_expert[u / kParts]] <= kBlockRows) continue;
    const long long row = (long long)u * kHeavyRows + warp * 2;
    const int s0 = row_slot[row], s1 = row_slot[row + 1];
    const __nv_bfloat16 *src0 = x + (long long)(s0 < 0 ? 0 : s0 / k) * d, *src1 = x + (long long)(s1 < 0 ? 0 : s1 / k) * d;
    const uint4 zero = make_uint4(0, 0, 0, 0);
#pragma unroll 4
    for (int c = lane * 8; c < d; c += 256) {
      const uint4 v0 = ld_nc_v4(src0 + c), v1 = ld_nc_v4(src1 + c);
      st_v4(out + row * d + c, s0 < 0 ? zero : v0);
      st_v4(out + (row + 1) * d + c, s1 < 0 ? zero : v1);
    }
  }
}

// smallest supported VPL in {1,2,4,8,16} covering the row, or 0
inline int pick_vpl(int d, int elem_bytes) {
  const long long row_bytes = (long long)d * elem_bytes;
  if (row_bytes % 16 != 0) return 0;
  const long long nvec = row_bytes / 16;
  for (int v = 1; v <= 16; v *= 2)
    if (nvec <= (long long)v * kWarp) return v;
  return 0;
}

#define LEWI_DISPATCH_VPL(VPL_VALUE, ...)        \
  switch (VPL_VALUE) {                           \
    case 1: { constexpr int VPL = 1; __VA_ARGS__; } break;   \
    case 2: { constexpr int VPL = 2; __VA_ARGS__; } break;   \
    case 4: { constexpr int VPL = 4; __VA_ARGS__; } break;   \
    case 8: { constexpr int VPL = 8; __VA_ARGS__; } break;   \
    default: { constexpr int VPL = 16; __VA_ARGS__; } break; \
  }

}  // namespace lewi
